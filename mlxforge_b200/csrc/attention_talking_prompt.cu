// Attention with talking heads for portions of prompts on the 5th-generation tensor cores: 8 or 16 query heads, four to a key head, keys
// and values of 128 channels, bfloat16.  The formulas are those of attention_talking.cu.
//
// The heads of a (query, key) pair meet before the softmax, so a block owns 16 queries with ALL heads and walks over the keys in tiles
// of 128 that start at multiples of 128 (a row's sums depend on positions only).  Both products stand on their heads: a KEY is a lane of
// tensor memory, a query and head a column,
//
//   S^T = K Q^T      per key head 128 keys x 64 (16 queries of its four heads), 32-bit in tensor memory
//   O^T += V^T P^T   128 channels x 64, the values read along their channels, P^T from shared memory
//
// because then the scores of one query and key over all heads can be in ONE thread: the columns of eight neighbours are two heads of
// four queries, and the load of 16 lanes x 16 columns gives a thread two of the heads of one query at four keys; over the key heads it
// has all of them.  The mixing s'_h = sum_g talk[h, g] s_g is then 32-bit multiply-adds on registers, two keys an instruction, with the
// matrix, every number twice, in shared memory (a load that all lanes share costs one pass).  Every head's own score is added last, so
// that a sum is rounded at its full size once or twice and not 16 times.
//
//   warps 0, 2, 3  keys and values by tensor copies (four pages that follow one another at once) into a ring of 16 KB stages
//   warp 1      both products: S of the next tile as soon as the scores are in registers, then O += V^T P^T
//   warps 4-11  two groups of four; a group's warps are the 128 keys, a group takes four queries at a time, twice a tile: soft cap, mixing,
//               mask, maxima (over a thread's keys, then lanes, then the group's warps by atomics), weights to shared memory, sums.  The
//               reference of a row is its running maximum, so that its largest weight is a 1 that bfloat16 holds exactly; rows of O
//               (columns of tensor memory) are multiplied where a maximum has moved.
//
// Keys are cut at multiples of 1024 where a query sees more; a block whose range is one cut writes its result itself, the others their
// sums for the merge of attention_talking_tc.cu.  Blocks with the most keys first.
//
// What bounds it: the softmax warps' own chain, two of them a scheduler.  Counters: no pipe is full (issue slots 38 %, special functions 23, FMA 18,
// integer 19, tensor 9); they wait for fixed latencies, tensor memory and barriers, a tenth of the time for instructions, as a loop over
// tiles is larger than the SM's instruction cache.  16 heads, one prompt of 2,048 tokens in one chunk, with its merge: 215
// (mma.sync, tiles of 32 keys) -> 111 us.  Measured on the way, at 113 us: the loop over a product's stages unrolled 122; so, and 1,024 single multiply-adds
// instead of 512 of pairs 133, with the matrix in the constant bank 130; four groups, a reference that moves only by 2^8 and no scores kept
// 125, but results 3 % further from 64 bits; cuts of 512 keys 153; products sent inside `if (lane == 0)` left the tile waiting for them
// (1,000 cycles a stage beside warps that are busy with multiply-adds, 400 as they are sent now).  Results are 1.4 % further from 64 bits than
// the other kernel's there (2.004e-3 of their norm, 1.976e-3): nothing is held in fewer bits, but a row's maximum, whose weight of 1 is not
// rounded, is taken anew every 128 keys instead of 32 and in every cut of 1,024 instead of 512.
#include <type_traits>

#include "attention_talking_prompt.cuh"
#include "common.cuh"
#include "tcgen05.cuh"
#include "tma_host.cuh"

namespace {

using namespace tc5;

constexpr int QT = 16, KT = 128, DIM = 128, CUT = 1024, STAGE = 16384, BOX = 16 * 128, SOFT = 8, THREADS = 32 * (SOFT + 4);
// of 168 registers a thread at launch: 128 x 56 + 256 x 224 = 384 x 168
constexpr int REGS_LESS = 56, REGS_MORE = 224, REGS_ALL = 128 * REGS_LESS + 32 * SOFT * REGS_MORE;
constexpr float LOG2E = 1.4426950408889634f;

struct Args {
  const __nv_bfloat16* q;
  __nv_bfloat16* out;
  const int* seq_q_start;
  const int* seq_q_len;
  const int* seq_ctx_len;
  const int* block_table;
  const float* talk;        // [heads, heads], or null: heads stay apart
  int table_row0, bt_stride, page_size;
  float scale, softcap;
  int window, chunk;
  int cuts;                 // 1: a block walks all its keys
  int from_keys;            // sequences whose queries see fewer keys are left out
  float* part_o;            // [rows, cuts, heads, 128]
  float* part_ml;           // [rows, cuts, heads, 2]: reference in powers of two and sum; sum -1: the row is done
  int* status;
};

__host__ __device__ constexpr int ring(int nh) { return nh == 16 ? 5 : 8; }
__host__ __device__ constexpr int used_smem(int nh) {
  return 2 * (nh / 4) * STAGE + ring(nh) * STAGE + nh * nh * 8 + 2 * QT * nh * 4 + (2 * ring(nh) + 4) * 8 + 16;
}

__device__ __forceinline__ float exp2_(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// numbers whose order as integers is that of the floats
__device__ __forceinline__ int ordered(float x) {
  const int i = __float_as_int(x);
  return i ^ (i >> 31 & 0x7fffffff);
}
__device__ __forceinline__ float unordered(int i) { return __int_as_float(i ^ (i >> 31 & 0x7fffffff)); }
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;\n" ::"r"(1 + group) : "memory"); }
__device__ __forceinline__ bool group_any(int group, bool x) {
  uint32_t r;
  asm volatile(
      "{\n.reg .pred p, q;\n"
      "setp.ne.u32 p, %2, 0;\n"
      "bar.red.or.pred q, %1, 128, p;\n"
      "selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r) : "r"(1 + group), "r"((uint32_t)x) : "memory");
  return r != 0;
}

// the softmax warps and the issuing ones: queries and matrix are in place
__device__ __forceinline__ void ready_sync() { asm volatile("bar.sync 5, %0;\n" ::"n"(32 * (SOFT + 1)) : "memory"); }

template <int NH, bool MIXED, bool CAP>
__global__ void __launch_bounds__(THREADS, 1)
talking_prompt_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_k4, const __grid_constant__ CUtensorMap map_v4, const Args a) {
  constexpr int G = NH / 4, RING = ring(NH), COLS = 2 * NH * QT;
  constexpr uint32_t O_COL = NH * QT;
  extern __shared__ __align__(1024) unsigned char smem[];
  // A tile is 16 positions from a multiple of 16 on: none has one key more than a tile of keys, or keys of two chunks (where the chunks' size is a
  // multiple too; keys are cut by that).  Short portions that so have a tile more, and stay in their chunk, have their first tile begin with
  // them: 60 of 30 tokens over 300 others are 120 blocks then and not 180 on 148 SMs, 43 us instead of 70, with chunks of 256 25 instead of 42.  Of
  // longer ones it is a smaller part and keys that straddle cost as much: 300 tokens over 1,001 others 92 us as it is, 95 from their first on.  The
  // heaviest blocks first: of the last queries all cuts, then of the queries before them.
  const int seq = blockIdx.y, q_len = a.seq_q_len[seq], ctx = a.seq_ctx_len[seq], begin = ctx - q_len;
  int lead = begin & (QT - 1);
  if (q_len <= 4 * QT && (lead + q_len + QT - 1) / QT > (q_len + QT - 1) / QT && (a.chunk == 0 || begin / a.chunk == (ctx - 1) / a.chunk)) lead = 0;
  const int tile = (lead + q_len + QT - 1) / QT - 1 - (int)blockIdx.x / a.cuts, cut = (int)blockIdx.x % a.cuts;
  if (tile < 0 || q_len == 0) return;
  const int row0 = max(0, tile * QT - lead), rows = min(q_len, tile * QT + QT - lead) - row0;
  const int q_start = a.seq_q_start[seq], pos0 = ctx - q_len + row0, pos_last = pos0 + rows - 1;
  // warps 0-3 copy and issue: the lowest come first where several warps are ready, and these have few instructions
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto first_of = [&](int pos) {
    int first = 0;
    if (a.window > 0) first = max(first, pos - a.window + 1);
    if (a.chunk > 0) first = max(first, pos / a.chunk * a.chunk);
    return first;
  };
  const int lo0 = first_of(pos0);                 // no query of the tile sees a key before it
  int k_first = lo0, k_last = pos_last;
  const bool alone = lo0 / CUT == pos_last / CUT || a.cuts == 1;
  if (a.cuts > 1) {
    k_first = max(lo0, (lo0 / CUT + cut) * CUT);
    k_last = min(pos_last, (lo0 / CUT + cut) * CUT + CUT - 1);
  }
  const long long slot0 = ((long long)(q_start + row0) * a.cuts + cut) * NH, slot_row = (long long)a.cuts * NH;
  if (talking_prompt_keys(ctx, a.window, a.chunk) < a.from_keys) {      // the other kernel's: its rows are done without a merge
    for (int i = tid; i < rows * NH && a.cuts > 1 && cut == 0; i += THREADS)
      *reinterpret_cast<float2*>(a.part_ml + (slot0 + i / NH * slot_row + i % NH) * 2) = make_float2(-INFINITY, -1.f);
    return;
  }
  if (k_first > k_last) {                         // a cut without keys: its rows are not read
    for (int i = tid; i < rows * NH; i += THREADS)
      *reinterpret_cast<float2*>(a.part_ml + (slot0 + i / NH * slot_row + i % NH) * 2) = make_float2(-INFINITY, 0.f);
    return;
  }
  const int kt0 = k_first / KT, n_tiles = k_last / KT - kt0 + 1;

  const uint32_t q_u = smem_u32(smem), p_u = q_u + G * STAGE, ring_u = p_u + G * STAGE, m_u = ring_u + RING * STAGE;
  const uint32_t talk_u = m_u + 2 * QT * NH * 4, alpha_u = m_u + QT * NH * 4;   // [query][head]: running maxima (as ordered integers); what older sums are multiplied with
  const uint32_t full0 = talk_u + NH * NH * 8, empty0 = full0 + 8 * RING, s_full = empty0 + 8 * RING, s_free = s_full + 8,
                 p_full = s_free + 8, o_done = p_full + 8, tmem_slot = o_done + 8;
  if (q_u & 1023u) {                              // never seen; refused rather than computed wrongly
    if (tid == 0 && a.status) atomicExch(a.status, 93);
    return;
  }
  bool dead = false;                              // a wait ran out: the rest of the block's waits are skipped
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    if (!dead && !mbar_wait(bar, parity, a.status, code)) dead = true;
  };

  if (tid == 0) {
    for (int i = 0; i < RING; i++) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, SOFT);
    mbar_init(p_full, SOFT);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, COLS);
  // Lines of a stage that no query sees can hold anything: the page's bits behind a sequence's end, or, where a granule was not fetched,
  // keys or values of any key head that stood there before.  Of keys they are scores that the mask takes away.  Of values, whose weight of
  // zero would not take away what is not finite, granules that were not fetched are no part of the product and the lines of fetched ones
  // are cleared behind the copy.
  __syncthreads();

  // a part of the launch's registers goes to the softmax warps
  if (warp < 4) regs_less<REGS_LESS>();
  if (warp == 0 || warp == 2 || warp == 3) {
    // ------------------------------------------------------------ producers: K of tile 0, then K of tile n + 1 and V of tile n, a stage in three each
    int turn = warp == 0 ? 0 : warp - 1;          // stages until this warp's next one
    const int* table = a.block_table + (long long)(a.table_row0 + seq) * a.bt_stride;
    const int gran = lane & 7, gi = lane & 3;
    auto page_of = [&](int n) {       // of a granule of 16 keys a lane; -1: no query sees one of them
      const int key16 = (kt0 + n) * KT + gran * 16;
      return n < n_tiles && key16 <= pos_last && key16 + 15 >= lo0 ? table[a.page_size == 16 ? key16 >> 4 : key16 / a.page_size] : -1;
    };
    int st = 0;
    uint32_t phase = 1;               // of the stage's release; a first use passes
    // a stage is two boxes of 64 keys x 64 channels: of keys one span of channels of all 128, of values both spans of 64 keys
    auto load = [&](int n, int page, bool values) {
#pragma unroll 1
      for (int part = 0; part < 2; part++) {
        const int g = values ? part * 4 + gi : gran;
        const int pg = __shfl_sync(0xffffffffu, page, g);
        const bool valid = pg >= 0;
        const int first = __shfl_sync(0xffffffffu, pg, lane & ~3);
        const uint32_t follows = __ballot_sync(0xffffffffu, a.page_size == 16 && valid && first >= 0 && pg == first + gi);
        const bool run0 = (follows & 15) == 15, run1 = (follows >> 4 & 15) == 15;
        const int page0 = __shfl_sync(0xffffffffu, pg, 0), page1 = __shfl_sync(0xffffffffu, pg, 4);
        const uint32_t bytes = __popc(__ballot_sync(0xffffffffu, valid) & 255u) * BOX;
        const int key16 = (kt0 + n) * KT + g * 16, in_page = a.page_size == 16 ? 0 : key16 % a.page_size;
        const bool single = valid && lane < 8 && !(lane < 4 ? run0 : run1);
        const int ch0 = values ? 0 : part * 64, ch1 = values ? 64 : part * 64;
#pragma unroll 1
        for (int kv = 0; kv < G; kv++) {
          if (turn-- > 0) {
            if (++st == RING) st = 0, phase ^= 1;
            continue;
          }
          turn = 2;
          const uint32_t bar = full0 + 8 * st, dst = ring_u + st * STAGE;
          wait(empty0 + 8 * st, phase, 94);
          expect_tx_one(bar, bytes);
          if (run0) tma_load_3d_one(dst, values ? &map_v4 : &map_k4, ch0, kv * 16, page0, bar);
          if (run1) tma_load_3d_one(dst + 8192, values ? &map_v4 : &map_k4, ch1, kv * 16, page1, bar);
          __syncwarp();
          if (single)                 // a granule of 16 lines a lane
            tma_load_2d(dst + lane * BOX, values ? &map_v : &map_k, lane < 4 ? ch0 : ch1, (pg * G + kv) * a.page_size + in_page, bar);
          __syncwarp();
          if (++st == RING) st = 0, phase ^= 1;
        }
      }
    };
    int now = page_of(0), next = page_of(1);
    load(0, now, false);
    for (int n = 0; n < n_tiles; n++) {
      const int after = page_of(n + 2);
      if (n + 1 < n_tiles) load(n + 1, next, false);
      load(n, now, true);
      now = next;
      next = after;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ both products
    ready_sync();
    fence_after();
    const uint32_t tmem = uniform(*reinterpret_cast<const uint32_t*>(smem + (tmem_slot - q_u)));
    int st = 0;
    uint32_t phase = 0;
    const unsigned long long ring_d = smem_desc(ring_u, 8192), q_d = smem_desc(q_u), p_d = smem_desc(p_u);
    // S of tile n, or O += V^T P^T: a stage is four steps of 16 for one key head
    auto product = [&](int n, auto what) {
      constexpr bool values = decltype(what)::value;
      constexpr uint32_t desc = bf16_idesc(128, 64, values, values), step = (values ? 2048 : 32) >> 4;
      const int key0 = (kt0 + n) * KT;
      const bool ragged = values && (key0 < lo0 || key0 + KT - 1 > pos_last);
      auto operands = [&](int part, int kv, unsigned long long& da, unsigned long long& db) {
        da = ring_d + (uint32_t)(st * (STAGE >> 4)), db = (values ? p_d : q_d) + (uint32_t)(kv * (STAGE >> 4) + part * (8192 >> 4));
        return tmem + (values ? O_COL : 0) + kv * 64;
      };
      auto stage = [&](int part, int kv) {
        fence_after();
        unsigned long long da, db;
        const uint32_t d = operands(part, kv, da, db);
        umma(d, da, db, desc, part > 0 ? 1u : (values && n > 0 ? 1u : 0u));
#pragma unroll
        for (uint32_t k = 1; k < 4; k++) umma(d, da + k * step, db + k * step, desc, 1u);
        umma_commit(empty0 + 8 * st);
      };
      if (ragged) {                   // the granules that were fetched, without their lines that no query sees
        const int first = max(0, (lo0 - key0) >> 4), last = min(7, (pos_last - key0) >> 4);
#pragma unroll 1
        for (int i = 0; i < 2 * G; i++) {
          wait(full0 + 8 * st, phase, 98);
          const int part = i / G;
#pragma unroll 1
          for (int at = lane; at < 32 * 8; at += 32) {
            const int r = at >> 3, key = r < 16 ? (lo0 & ~15) + r : (pos_last & ~15) + r - 16, line = key - key0 - part * 64;
            if ((r < 16 ? key >= lo0 : key <= pos_last) || line < 0 || line >= 64) continue;
            uint4* const to = reinterpret_cast<uint4*>(smem + (ring_u - q_u) + st * STAGE + line * 128 + (at & 7) * 16);
            to[0] = to[8192 / 16] = make_uint4(0, 0, 0, 0);
          }
          fence_proxy();
          __syncwarp();
          fence_after();
          unsigned long long da, db;
          const uint32_t d = operands(part, i % G, da, db);
#pragma unroll 1
          for (int k = max(0, first - part * 4); k <= min(3, last - part * 4); k++)
            umma(d, da + k * step, db + k * step, desc, n > 0 || part * 4 + k > first ? 1u : 0u);
          umma_commit(empty0 + 8 * st);
          if (++st == RING) st = 0, phase ^= 1;
        }
      } else {                        // the next stage's barrier is looked at before this one's products are sent: its answer takes as long as two
        bool there = mbar_peek(full0 + 8 * st, phase);
#pragma unroll 1
        for (int i = 0; i < 2 * G; i++) {
          if (!there) wait(full0 + 8 * st, phase, values ? 98 : 95);
          const int next = st + 1 == RING ? 0 : st + 1;
          const uint32_t next_phase = st + 1 == RING ? phase ^ 1 : phase;
          if (i + 1 < 2 * G) there = mbar_peek(full0 + 8 * next, next_phase);
          stage(i / G, i % G);
          st = next, phase = next_phase;
        }
      }
      umma_commit(values ? o_done : s_full);
    };
    product(0, std::false_type());
#pragma unroll 1
    for (int n = 0; n < n_tiles; n++) {
      if (n + 1 < n_tiles) {
        wait(s_free, n & 1, 96);
        product(n + 1, std::false_type());
      }
      wait(p_full, n & 1, 97);
      product(n, std::true_type());
    }
    __syncwarp();
  } else if (warp >= 4) {
    regs_more<REGS_MORE>();
    const int st_id = tid - 128;           // among the softmax threads
    for (int i = st_id; i < QT * NH; i += 32 * SOFT) reinterpret_cast<int*>(smem + (m_u - q_u))[i] = ordered(-INFINITY);
    if (MIXED)                        // every number twice
      for (int i = st_id; i < NH * NH; i += 32 * SOFT) {
        const float t = a.talk[i];
        reinterpret_cast<float2*>(smem + (talk_u - q_u))[i] = make_float2(t, t);
      }
    constexpr int PIECES = QT * NH * (DIM / 8) / (32 * SOFT);
    uint4 qv[PIECES];
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
      const int at = i * 32 * SOFT + st_id, r = at / (DIM / 8 * NH);
      qv[i] = make_uint4(0, 0, 0, 0);
      if (r < rows) qv[i] = *reinterpret_cast<const uint4*>(a.q + (long long)(q_start + row0) * NH * DIM + at * 8);
    }
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
      const int at = i * 32 * SOFT + st_id, piece = at % (DIM / 8), h = at / (DIM / 8) % NH, r = at / (DIM / 8 * NH), hl = h & 3;
      const int n = (2 * (r >> 2) + (hl >> 1)) * 8 + 2 * (r & 3) + (hl & 1);
      *reinterpret_cast<uint4*>(smem + (h >> 2) * STAGE + (piece >> 3) * 8192 + n * 128 + (((piece & 7) ^ (n & 7)) << 4)) = qv[i];
    }
    fence_proxy();
    fence_before();
    ready_sync();
    fence_after();
    const uint32_t tmem = *reinterpret_cast<const uint32_t*>(smem + (tmem_slot - q_u));
    // ------------------------------------------------------------ soft cap, mixing, softmax
    // a group of four warps has the queries 4 group + qq, then 8 + 4 group + qq
    const int group = (warp >> 2) - 1, wq = warp & 3, qq = lane & 3, k8 = lane >> 2;
    const bool upper = lane & 16;
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    const float cap = a.softcap, pre = CAP ? a.scale / cap * (2.0f * LOG2E) : a.scale;
    const f32x2 pre2 = pack2(pre, pre), cap2 = pack2(cap, cap), ncap2 = pack2(-cap, -cap), one2 = pack2(1.f, 1.f), log2e2 = pack2(LOG2E, LOG2E);
    int* const most = reinterpret_cast<int*>(smem + (m_u - q_u));
    float* const alpha = reinterpret_cast<float*>(smem + (alpha_u - q_u));
    // of the query's heads a lane keeps the sums of own, own + 8: its bits 16, 8, 4 choose halves
    constexpr int OWN = NH / 8;
    const int own = ((lane & 16) ? 1 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 4 : 0);
    float l[2][OWN], before[2] = {-INFINITY, -INFINITY};      // before: row and head 4 qb + (tid & 127) / NH, (tid & 127) % NH
#pragma unroll
    for (int i = 0; i < OWN; i++) l[0][i] = l[1][i] = 0.f;
    // over the lanes with one query: numbers of NH heads down to OWN, half of the heads a step
    auto over_lanes = [&](float (&x)[NH], auto join) {
#pragma unroll
      for (int i = 0; i < NH / 2; i++) {
        const float give = upper ? x[2 * i] : x[2 * i + 1], keep = upper ? x[2 * i + 1] : x[2 * i];
        x[i] = join(keep, __shfl_xor_sync(0xffffffffu, give, 16));
      }
#pragma unroll
      for (int i = 0; i < NH / 4; i++) {
        const float give = (lane & 8) ? x[2 * i] : x[2 * i + 1], keep = (lane & 8) ? x[2 * i + 1] : x[2 * i];
        x[i] = join(keep, __shfl_xor_sync(0xffffffffu, give, 8));
      }
#pragma unroll
      for (int i = 0; i < OWN; i++) {
        const float give = (lane & 4) ? x[2 * i] : x[2 * i + 1], keep = (lane & 4) ? x[2 * i + 1] : x[2 * i];
        x[i] = join(keep, __shfl_xor_sync(0xffffffffu, give, 4));
      }
    };

#pragma unroll 1
    for (int n = 0; n < n_tiles; n++) {
      const int key0 = (kt0 + n) * KT, key = key0 + wq * 32 + k8;
      const bool edge = key0 + KT - 1 > pos0 || key0 < first_of(pos_last);
      wait(s_full, n & 1, 99);
      fence_after();
#pragma unroll 1
      for (int qi = 0; qi < 2; qi++) {
        const int qb = 2 * qi + group, at = (4 * qb + qq) * NH;
        const bool some = 4 * qb < rows;
        // the scores of all heads at this thread's four keys 32 wq + k8 + 8 j; a piece of 16 keys and four heads is on its way while the one
        // before is worked on
        f32x2 s[NH][2];                 // keys j = 0, 1 and 2, 3
        if (some) {
          uint32_t u[2][8];
          const uint32_t from = tmem + lanes + qb * 16;
          tmem_ld_16x16_issue(from, u[0]);
#pragma unroll
          for (int i = 0; i < 2 * G; i++) {
            const int kv = i >> 1, half = i & 1;
            uint32_t(&w)[8] = u[i & 1];
            tmem_landed(w);
            if (i + 1 < 2 * G) tmem_ld_16x16_issue(from + ((uint32_t)((i + 1 & 1) * 16) << 16) + (i + 1 >> 1) * 64, u[i + 1 & 1]);
#pragma unroll
            for (int p = 0; p < 2; p++) {       // a pair of heads
              const f32x2 v0 = mul2(pack2(__uint_as_float(w[4 * p]), __uint_as_float(w[4 * p + 2])), pre2);
              const f32x2 v1 = mul2(pack2(__uint_as_float(w[4 * p + 1]), __uint_as_float(w[4 * p + 3])), pre2);
              f32x2& s0 = s[kv * 4 + 2 * p][half];
              f32x2& s1 = s[kv * 4 + 2 * p + 1][half];
              s0 = v0, s1 = v1;
              if (CAP) {
                // with v = 2 log2(e) x: cap tanh(x) = cap (1 - 2^-|v|) / (1 + 2^-|v|)
                const float2 a0 = unpack2(v0), a1 = unpack2(v1);
                const f32x2 t0 = pack2(exp2_(-fabsf(a0.x)), exp2_(-fabsf(a0.y))), t1 = pack2(exp2_(-fabsf(a1.x)), exp2_(-fabsf(a1.y)));
                const f32x2 d0 = fma2(t0, one2, one2), d1 = fma2(t1, one2, one2);
                f32x2 y0 = fma2(t0, ncap2, cap2), y1 = fma2(t1, ncap2, cap2);
                if (MIXED) {                    // one reciprocal for two heads that meet anyway
                  const float2 d = unpack2(mul2(d0, d1));
                  const f32x2 r = pack2(rcp_(d.x), rcp_(d.y));
                  y0 = mul2(y0, mul2(r, d1)), y1 = mul2(y1, mul2(r, d0));
                } else {
                  const float2 e0 = unpack2(d0), e1 = unpack2(d1);
                  y0 = mul2(y0, pack2(rcp_(e0.x), rcp_(e0.y))), y1 = mul2(y1, pack2(rcp_(e1.x), rcp_(e1.y)));
                }
                const float2 b0 = unpack2(y0), b1 = unpack2(y1);
                s0 = pack2(copysignf(b0.x, a0.x), copysignf(b0.y, a0.y)), s1 = pack2(copysignf(b1.x, a1.x), copysignf(b1.y, a1.y));
              }
            }
          }
        }
        if (qi == 1) {
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_free);
        }
        if (!some) continue;
        // mixed: the other key heads' heads in turn, a head's own four last, of them its own pair, and in it the head itself (a sum is
        // rounded at its full size once the head's own score is in it)
        f32x2 x[NH][2];
        float by[NH];
        uint32_t talk_here;              // a new number to the compiler: else it loads the matrix once for all tiles, and spills it
        asm volatile("mov.u32 %0, %1;" : "=r"(talk_here) : "r"(talk_u));
#pragma unroll
        for (int h = 0; h < NH; h++) {
          if (MIXED) {
#pragma unroll
            for (int i = 0; i < NH; i += 2) {
              const int q = (h / 4 + 1 + i / 4) % G * 4, g = q + (q == h / 4 * 4 ? (i & 2) ^ (h & 2) ^ 2 : i & 2);      // a pair of heads
              const int ga = q == h / 4 * 4 && (h & 2) == (g & 2) && !(h & 1) ? g + 1 : g, gb = ga ^ 1;
              f32x2 t0, t1;
              asm("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(t0), "=l"(t1) : "r"(talk_here + (h * NH + g) * 8));
#pragma unroll
              for (int j = 0; j < 2; j++) {
                x[h][j] = i == 0 ? mul2(ga == g ? t0 : t1, s[ga][j]) : fma2(ga == g ? t0 : t1, s[ga][j], x[h][j]);
                x[h][j] = fma2(ga == g ? t1 : t0, s[gb][j], x[h][j]);
              }
            }
          } else {
            x[h][0] = s[h][0], x[h][1] = s[h][1];
          }
        }
        if (edge) {
          const int pos = pos0 + 4 * qb + qq, first = first_of(pos);
          bool seen[4];
#pragma unroll
          for (int j = 0; j < 4; j++) seen[j] = key + 8 * j <= pos && key + 8 * j >= first;
#pragma unroll
          for (int h = 0; h < NH; h++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
              const float2 y = unpack2(x[h][j]);
              x[h][j] = pack2(seen[2 * j] ? y.x : -INFINITY, seen[2 * j + 1] ? y.y : -INFINITY);
            }
        }
        // ---- maxima: over the thread's keys, the lanes with this query, the group's warps
#pragma unroll
        for (int h = 0; h < NH; h++) {
          const float2 y = unpack2(x[h][0]), z = unpack2(x[h][1]);
          by[h] = fmaxf(max3(y.x, y.y, z.x), z.y);
        }
        over_lanes(by, [](float p, float q) { return fmaxf(p, q); });
#pragma unroll
        for (int i = 0; i < OWN; i++) atomicMax(most + at + own + 8 * i, ordered(by[i]));
        group_sync(group);
        bool moved = false;
        if ((tid & 127) < 4 * NH) {
          // a maximum in powers of two, rounded once: weights, moved sums and the merge go by this number
          const int i = 4 * qb * NH + (tid & 127);
          const float m = unordered(most[i]), f = m == -INFINITY ? 1.f : exp2_(__fmul_rn(qi ? before[1] : before[0], LOG2E) - __fmul_rn(m, LOG2E));
          moved = f != 1.f;
          alpha[i] = f;
          if (qi) before[1] = m;
          else before[0] = m;
        }
        // ---- weights
        if (n > 0) wait(o_done, (n - 1) & 1, 100);           // P of the tile before has been read
        // P^T along N, [key head][128 keys][64: query * 4 + head]
        const uint32_t p_at = p_u + (wq * 32 + k8) * 128 + (((uint32_t)(2 * qb + (qq >> 1)) ^ (uint32_t)k8) << 4) + (qq & 1) * 8;
#pragma unroll
        for (int kv = 0; kv < G; kv++) {
          const int4 o4 = *reinterpret_cast<const int4*>(most + at + kv * 4);
          const int oi[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int h = kv * 4 + e;
            const float m = unordered(oi[e]), off = m == -INFINITY ? 0.f : __fmul_rn(m, LOG2E);
            const f32x2 off2 = pack2(-off, -off);
#pragma unroll
            for (int j = 0; j < 2; j++) {
              const float2 y = unpack2(fma2(x[h][j], log2e2, off2));
              x[h][j] = pack2(exp2_(y.x), exp2_(y.y));
            }
            const float2 y = unpack2(x[h][0]), z = unpack2(x[h][1]);
            by[h] = (y.x + y.y) + (z.x + z.y);
          }
#pragma unroll
          for (int j = 0; j < 4; j++) {
            auto of = [&](int e) { return j & 1 ? unpack2(x[kv * 4 + e][j >> 1]).y : unpack2(x[kv * 4 + e][j >> 1]).x; };
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};\n" ::"r"(p_at + kv * STAGE + j * 1024), "r"(pack_bf16(of(0), of(1))), "r"(pack_bf16(of(2), of(3)))
                         : "memory");
          }
        }
        over_lanes(by, [](float p, float q) { return p + q; });
        // ---- older sums of rows whose maximum has moved
        if (group_any(group, moved) && n > 0) {
          fence_after();
#pragma unroll
          for (int i = 0; i < OWN; i++) {
            const float f = alpha[at + own + 8 * i];
            if (qi) l[1][i] *= f;
            else l[0][i] *= f;
          }
#pragma unroll 1
          for (int kv = 0; kv < G; kv++) {
            uint32_t o[16];
            tmem_ld16_issue(tmem + lanes + O_COL + kv * 64 + qb * 16, o);
            tmem_landed(o);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const float4 f = *reinterpret_cast<const float4*>(alpha + (4 * qb + i) * NH + kv * 4);
              o[4 * i] = __float_as_uint(__uint_as_float(o[4 * i]) * f.x);
              o[4 * i + 1] = __float_as_uint(__uint_as_float(o[4 * i + 1]) * f.y);
              o[4 * i + 2] = __float_as_uint(__uint_as_float(o[4 * i + 2]) * f.z);
              o[4 * i + 3] = __float_as_uint(__uint_as_float(o[4 * i + 3]) * f.w);
            }
            tmem_st16(tmem + lanes + O_COL + kv * 64 + qb * 16, o);
          }
          tmem_wait_st();
        }
#pragma unroll
        for (int i = 0; i < OWN; i++) {
          if (qi) l[1][i] += by[i];
          else l[0][i] += by[i];
        }
      }
      // a group without queries must not arrive for the next tile while the other works on this
      if (n > 0) wait(o_done, (n - 1) & 1, 103);
      fence_proxy();          // P, before the product reads it
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }

    // ---- sums over the group's warps, where the queries stood: [query block][warp][query][head], then [query][head]
    wait(o_done, (n_tiles - 1) & 1, 102);
    fence_after();
    float* const part = reinterpret_cast<float*>(smem);
    float* const sums = part + 64 * NH;
#pragma unroll
    for (int qi = 0; qi < 2; qi++)
#pragma unroll
      for (int i = 0; i < OWN; i++) part[(((2 * qi + group) * 4 + wq) * 4 + qq) * NH + own + 8 * i] = l[qi][i];
    group_sync(group);
    for (int i = tid & 127; i < 8 * NH; i += 128) {
      const int qb = 2 * (i / (4 * NH)) + group, at = i % (4 * NH), r = 4 * qb + at / NH;
      const float* p = part + qb * 16 * NH + at;
      const float sum = (p[0] + p[4 * NH]) + (p[8 * NH] + p[12 * NH]), m = unordered(most[r * NH + at % NH]);
      sums[r * NH + at % NH] = 1.0f / sum;
      if (a.cuts > 1 && r < rows)
        *reinterpret_cast<float2*>(a.part_ml + (slot0 + r * slot_row + at % NH) * 2) =
            alone ? make_float2(-INFINITY, -1.f) : make_float2(m == -INFINITY ? -INFINITY : __fmul_rn(m, LOG2E), sum);
    }
    group_sync(group);
    const int ch = wq * 32 + lane;
#pragma unroll 1
    for (int qb = group; 4 * qb < rows; qb += 2)
#pragma unroll 1
      for (int kv = 0; kv < G; kv++) {
        uint32_t o[16];
        tmem_ld16_issue(tmem + lanes + O_COL + kv * 64 + qb * 16, o);
        tmem_landed(o);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = 4 * qb + i;
          if (r >= rows) break;
          const float4 f = *reinterpret_cast<const float4*>(sums + r * NH + kv * 4);
          const float by[4] = {f.x, f.y, f.z, f.w};
          if (alone) {
            __nv_bfloat16* const to = a.out + ((long long)(q_start + row0 + r) * NH + kv * 4) * DIM + ch;
#pragma unroll
            for (int h = 0; h < 4; h++) to[h * DIM] = __float2bfloat16_rn(__uint_as_float(o[4 * i + h]) * by[h]);
          } else {
            float* const to = a.part_o + (slot0 + r * slot_row + kv * 4) * DIM + ch;
#pragma unroll
            for (int h = 0; h < 4; h++) to[h * DIM] = __uint_as_float(o[4 * i + h]);
          }
        }
      }
  }
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc(*reinterpret_cast<const uint32_t*>(smem + (tmem_slot - q_u)), COLS);
  }
}

template <int NH, bool MIXED, bool CAP>
int launch(const void* k_pool, const void* v_pool, long long pool_rows, const Args& a, int n_seqs, int max_q_len, cudaStream_t stream) {
  CUtensorMap k, v;
  int rc = tma_host::bf16_map(k_pool, pool_rows, DIM, 16, 64, &k);
  if (rc == 0) rc = tma_host::bf16_map(v_pool, pool_rows, DIM, 16, 64, &v);
  if (rc) return rc;
  CUtensorMap k4 = k, v4 = v;
  if (a.page_size == 16) {
    const long long pages = pool_rows / (NH / 4 * 16);
    rc = tma_host::bf16_map_pages(k_pool, pages, NH / 4 * 16, DIM, 4, &k4);
    if (rc == 0) rc = tma_host::bf16_map_pages(v_pool, pages, NH / 4 * 16, DIM, 4, &v4);
    if (rc) return rc;
  }
  constexpr int bytes = used_smem(NH);
  static_assert(bytes <= 227 * 1024, "shared memory of a block");
  static DeviceOnce once;
  const int d = mf_current_device();
  if (d < 0) return MF_ERR_BAD_ARG;
  if (!once.done[d]) {
    cudaError_t e = cudaFuncSetAttribute(talking_prompt_kernel<NH, MIXED, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncAttributes built;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&built, talking_prompt_kernel<NH, MIXED, CAP>);
    if (e != cudaSuccess) return (int)e;
    if (built.numRegs * THREADS < REGS_ALL) return MF_ERR_BAD_ARG;        // built with fewer, the softmax warps would wait for theirs for good
    once.done[d] = true;
  }
  const dim3 grid((max_q_len + 2 * QT - 2) / QT * a.cuts, n_seqs);
  talking_prompt_kernel<NH, MIXED, CAP><<<grid, THREADS, bytes, stream>>>(k, v, k4, v4, a);
  return (int)cudaGetLastError();
}

}  // namespace

// The groupings that configurations use.  Heads of 64 would be half a stage wide and other groupings no 64 columns a key head: they need stages and
// products of another shape, which are not built.
bool talking_prompt_takes(int n_heads, int n_kv, int dim, int vdim, const void* q, const void* k_pool, const void* v_pool,
                          long long pool_rows) {
  return (n_heads == 16 || n_heads == 8) && n_heads == 4 * n_kv && dim == DIM && vdim == DIM && pool_rows > 0 &&
         !(((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15);
}

int talking_prompt_cuts(int splits, int chunk) {
  if (splits <= 1) return 1;
  if (chunk > 0 && chunk % CUT == 0) return min(splits, chunk / CUT);
  return chunk > 0 && CUT % chunk == 0 ? 1 : splits;
}

int talking_prompt_launch(const void* q, const void* k_pool, const void* v_pool, void* out, const int* seq_q_start, const int* seq_q_len,
                          const int* seq_ctx_len, int table_row0, int n_seqs, int max_q_len, int n_heads, const int* block_table, int bt_stride,
                          int page_size, long long pool_rows, float scale, float softcap, const float* talk, int window, int chunk, int cuts,
                          int from_keys, float* part_o, float* part_ml, int* status, cudaStream_t stream) {
  const Args a{(const __nv_bfloat16*)q, (__nv_bfloat16*)out, seq_q_start, seq_q_len, seq_ctx_len, block_table, talk, table_row0, bt_stride,
               page_size, scale, softcap, window, chunk, cuts, from_keys, part_o, part_ml, status};
  const auto go = [&](auto nh) {
    constexpr int NH = decltype(nh)::value;
    if (talk) return softcap > 0.f ? launch<NH, true, true>(k_pool, v_pool, pool_rows, a, n_seqs, max_q_len, stream)
                                   : launch<NH, true, false>(k_pool, v_pool, pool_rows, a, n_seqs, max_q_len, stream);
    return softcap > 0.f ? launch<NH, false, true>(k_pool, v_pool, pool_rows, a, n_seqs, max_q_len, stream)
                         : launch<NH, false, false>(k_pool, v_pool, pool_rows, a, n_seqs, max_q_len, stream);
  };
  return n_heads == 16 ? go(std::integral_constant<int, 16>()) : go(std::integral_constant<int, 8>());
}
