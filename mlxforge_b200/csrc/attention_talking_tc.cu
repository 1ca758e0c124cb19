// Attention with talking heads for portions of prompts, bfloat16, on the tensor cores (mma.sync): sizes that attention_talking_prompt.cu
// does not take, and its short sequences.
//
// The formulas are those of attention_talking.cu.  The mixing of the heads' scores before the
// softmax couples all heads of a (query, key) pair, so a block owns a tile of 16 queries of one
// sequence with ALL heads, one warp per head, and walks over the keys in tiles of 32 that start
// at multiples of 32 (the order of every sum depends on positions only).  Per key tile:
//
//   1. warp h:  S_h = Q_h K_g(h)^T (mma.sync m16n8k16, 32-bit accumulators), scale, soft cap,
//               stored to shared memory in 32-bit;
//   2. the heads mixed, s'_h = sum_g talk[h, g] s_g, as one 16 x 8 x 16 product per query and eight keys, and the mask
//               (causal, chunk, window, length), in place.  Both factors are cut into three bfloat16 pieces (3 x 8 bits:
//               all 24 of a 32-bit number) and the six products of pieces down to 2^-16 of the leading one are added in the
//               tensor core (off by 4.7e-8 of the mixed scores' root mean square, 16 32-bit multiply-adds by 7.4e-8),
//               the smallest first: what is left out is 2^-24 of a term, the rounding of a 32-bit multiplication;
//   3. warp h:  online softmax of its mixed scores (32-bit), P_h rounded to bfloat16 as the
//               A operand, O_h += P_h V_g(h).
//
// Keys and values of a tile come in by tensor copies (other head sizes than 64 and 128 by cp.async): the next tile's keys while heads
// are mixed and the softmax runs, its values while its own scores are made, so one buffer of each is enough and no step waits for
// memory.
//
// Decoding (one query per sequence) has a kernel of its own further down: the keys are cut into splits of
// TT_SPLIT_TILES tiles that start at multiples of that many tiles, a block per (sequence, split)
// writes its unnormalised output with its maximum and sum, and a merge kernel joins the
// splits.  A split's range depends on positions only.  Portions of prompts whose queries see more
// than TT_PREFILL_SPLIT_TILES tiles of keys are cut the same way (the last tile of queries of a
// long prompt would otherwise walk all its keys alone while the blocks of the first tiles are
// long done), the tiles with the most keys first.
//
// What bounds it: 1,400 mma.sync a tile (13 cycles each and scheduler, 4,700 of a tile's cycles), then the arithmetic beside them, in three
// phases that one block of 16 heads goes through together.  2,048 tokens of 16 / 4 heads of 128 in one chunk: 224 -> 202 us, 9,400 cycles
// a tile: its copies as cp.async, 64 KB through the warps' own load path, were 2,700 of 10,300 cycles by a block's clock, whether or
// not they looked pages up; the tensor copies need the products' addresses to fold (the head size as a constant), else
// their swizzle costs what they save (234 us).  Two score tiles and two barriers instead of three were no faster (247 us).
#include "attention_talking_prompt.cuh"
#include "common.cuh"
#include "tma_host.cuh"

#define TT_BM 16
#define TT_BN 32
#define TT_SPAD 4          // floats of padding per row of the score tile
#define TT_SPLIT_TILES 2   // key tiles per split when decoding (64 keys)
#define TT_PREFILL_SPLIT_TILES 32   // and for portions of prompts (1024 keys; half of that on lanes whose queries see at most
                                    // 4096: one prompt of 2,048 tokens then fills the SMs evenly, and the partial results,
                                    // a row of 32-bit outputs a split, stay few)

__device__ __forceinline__ void tt_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t tt_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tt_ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tt_ldmatrix_x4(uint32_t (&r)[4], const void* p) { tt_ldmatrix_x4(r, tt_addr(p)); }
__device__ __forceinline__ void tt_ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tt_ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) { tt_ldmatrix_x4_trans(r, tt_addr(p)); }
__device__ __forceinline__ void tt_cp_async16(void* smem, const void* gmem) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(addr), "l"(gmem) : "memory");
}
__device__ __forceinline__ void tt_cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void tt_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tt_wait(uint32_t bar, uint32_t parity, int* status, int code) {
  for (unsigned i = 0; i < 1u << 24; i++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return;
  }
  if (status) atomicExch(status, code);
}
__device__ __forceinline__ void tt_tensor_copy(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
template <int N>
__device__ __forceinline__ void tt_cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t tt_pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// two 32-bit numbers as three pairs of bfloat16 whose sums they are
__device__ __forceinline__ void tt_pieces(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    p[i] = tt_pack(x, y);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
#define TT_GRANULES (2 * (TT_PREFILL_SPLIT_TILES + 2))      // of 16 keys, the most of a block whose keys are cut
#define TT_LOG2E 1.4426950408889634f
// a maximum in powers of two, rounded once: the weights, what moves older sums to a new maximum and the merge of the splits all
// go by this number, so that its rounding (1e-3 of a weight at scores of 20,000) drops out
__device__ __forceinline__ float tt_max_log2(float m) { return __fmul_rn(m, TT_LOG2E); }
__device__ __forceinline__ float tt_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// tanh in 32-bit arithmetic through one exponential and one reciprocal: (1 - e^{-2|x|}) / (1 + e^{-2|x|})
__device__ __forceinline__ float tt_tanh(float x) {
  const float t = tt_exp2(-2.0f * TT_LOG2E * fabsf(x));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + t));
  return copysignf((1.0f - t) * r, x);
}

// register `reg` of the mixing matrix as A fragments of its three pieces, [piece][register][lane]: rows r0 (+ 8), columns c2 (+ 8)
// and the next, zero beyond H
__device__ __forceinline__ void tt_talk_pieces(const float* talk, int H, int reg, int lane, uint32_t* tk) {
  const int h = (lane >> 2) + (reg & 1) * 8, g = (lane & 3) * 2 + (reg >> 1) * 8;
  auto at = [&](int g) { return h < H && g < H ? (talk ? talk[h * H + g] : 0.f) : 0.f; };
  uint32_t p[3];
  tt_pieces(at(g), at(g + 1), p);
#pragma unroll
  for (int i = 0; i < 3; i++) tk[(i * 4 + reg) * 32 + lane] = p[i];
}
// c[heads r0 (+ 8), keys c2, c2 + 1] = the mixed scores of eight keys; `from` is head 0's score of key r0, heads head_ld apart
__device__ __forceinline__ void tt_mix(const uint32_t (&t)[3][4], const float* from, int head_ld, int H, int c2, float (&c)[4]) {
  auto score = [&](int g) { return g < H ? from[(size_t)g * head_ld] : 0.f; };
  uint32_t lo[3], hi[3];
  tt_pieces(score(c2), score(c2 + 1), lo);
  tt_pieces(score(c2 + 8), score(c2 + 9), hi);
  c[0] = c[1] = c[2] = c[3] = 0.f;
  tt_mma(c, t[2], lo[0], hi[0]);
  tt_mma(c, t[0], lo[2], hi[2]);
  tt_mma(c, t[1], lo[1], hi[1]);
  tt_mma(c, t[1], lo[0], hi[0]);
  tt_mma(c, t[0], lo[1], hi[1]);
  tt_mma(c, t[0], lo[0], hi[0]);
}

struct TtArgs {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k_pool;
  const __nv_bfloat16* v_pool;
  __nv_bfloat16* out;
  const int* seq_q_start;
  const int* seq_q_len;
  const int* seq_ctx_len;
  const int* block_table;
  const float* talk;
  int table_row0, bt_stride, page_size, n_heads, n_kv, dim;
  float scale, softcap;
  int window, chunk;
  int splits;               // 0: every block walks all its keys; else gridDim.z splits of split_tiles tiles
  int split_tiles;
  float* part_o;            // [rows, splits, H, VDIM] unnormalised outputs of the splits
  float* part_ml;           // [rows, splits, H, 2]    maximum (in powers of two) and sum
  int* status;              // codes 91 (keys) and 92 (values): a wait for a copy ran out
  long long pool_rows;      // rows (pages x KV heads x page size) of either pool
  int below_keys;           // > 0: sequences whose queries see as many keys are left out
};

// DIM: the head size, where keys and values come by tensor copies (64 or 128, and values of whole 64-wide spans), [head][span][32 keys]
// [128 bytes], 128-byte swizzle; 0: by cp.async in padded rows.
template <int VDIM, int MAXH, int DIM>
__global__ void __launch_bounds__(32 * MAXH)
talking_attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                            const TtArgs a) {
  extern __shared__ __align__(1024) unsigned char tt_smem[];
  constexpr bool TENSOR = DIM > 0;
  const int H = a.n_heads, G = a.n_kv, dim = TENSOR ? DIM : a.dim;
  const int rep = H / G;
  const int seq = blockIdx.y;
  const int q_len = a.seq_q_len[seq];
  const int tiles = (q_len + TT_BM - 1) / TT_BM;
  if ((int)blockIdx.x >= tiles) return;
  const int row0 = (tiles - 1 - (int)blockIdx.x) * TT_BM;       // the tiles with the most keys first
  const int q_start = a.seq_q_start[seq], ctx = a.seq_ctx_len[seq];
  if (a.below_keys > 0 && talking_prompt_keys(ctx, a.window, a.chunk) >= a.below_keys) return;
  const int pos0 = ctx - q_len + row0;                       // position of the tile's first query
  const int rows = min(TT_BM, q_len - row0);
  const int* table = a.block_table + (long long)(a.table_row0 + seq) * a.bt_stride;

  const int qs_ld = dim + 8, vs_ld = VDIM + 8;
  constexpr int sc_ld = TT_BN + TT_SPAD, sc_hd = TT_BM * sc_ld + 4;         // a head's rows: heads in other banks
  const int k_ld = TENSOR ? dim : qs_ld, v_ld = TENSOR ? VDIM : vs_ld;      // a key's share
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(tt_smem);           // [G][32][k_ld]
  __nv_bfloat16* Vs = Ks + (size_t)G * TT_BN * k_ld;                        // [G][32][v_ld]
  __nv_bfloat16* Qs = Vs + (size_t)G * TT_BN * v_ld;                        // [H][16][qs_ld]
  float* sc = reinterpret_cast<float*>(Qs + (size_t)H * TT_BM * qs_ld);     // [H][sc_hd]
  // the mixing matrix as A fragments of its three pieces: [piece][register][lane], zero beyond H
  uint32_t* tk = reinterpret_cast<uint32_t*>(sc + (size_t)H * sc_hd);

  const int tid = threadIdx.x, nthreads = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5;          // warp = head
  const int r0 = lane >> 2, c2 = (lane & 3) * 2;

  // queries of the tile, all heads: rows beyond the portion are zero
  const int dv8 = dim / 8;
  for (int i = tid; i < H * TT_BM * dv8; i += nthreads) {
    const int h = i / (TT_BM * dv8), rem = i - h * TT_BM * dv8;
    const int r = rem / dv8, c = (rem - r * dv8) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < rows) v = *reinterpret_cast<const uint4*>(a.q + ((long long)(q_start + row0 + r) * H + h) * dim + c);
    *reinterpret_cast<uint4*>(Qs + ((size_t)h * TT_BM + r) * qs_ld + c) = v;
  }
  __shared__ __align__(8) unsigned long long bars[2];      // the keys, the values of a tile are there
  const uint32_t k_full = tt_addr(bars), v_full = k_full + 8;
  if (TENSOR && tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(k_full));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(v_full));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __shared__ int first_s[TT_BM];       // the first key that each query sees
  if (tid < TT_BM) {
    const int pi = pos0 + tid;
    int first = 0;
    if (a.window > 0) first = max(first, pi - a.window + 1);
    if (a.chunk > 0) first = max(first, pi / a.chunk * a.chunk);
    first_s[tid] = first;
  }
  if (warp < 4) tt_talk_pieces(a.talk, H, warp, lane, tk);

  // the first key any query of the tile sees: that of its first query
  int lo0 = 0;
  if (a.window > 0) lo0 = max(lo0, pos0 - a.window + 1);
  if (a.chunk > 0) lo0 = max(lo0, pos0 / a.chunk * a.chunk);
  const int pos_last = pos0 + rows - 1;

  float o[VDIM / 8][4];
#pragma unroll
  for (int i = 0; i < VDIM / 8; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  const int g_own = warp / rep;
  const bool has_head = warp < H;

  int k_first = (lo0 / TT_BN) * TT_BN, k_last = pos_last;
  if (a.splits > 0) {      // this block's share: tiles [z, z + 1) * TT_SPLIT_TILES of the sequence
    const int span = a.split_tiles * TT_BN;
    const int first_split = k_first / span;
    k_first = max(k_first, (first_split + (int)blockIdx.z) * span);
    k_last = min(k_last, (first_split + (int)blockIdx.z + 1) * span - 1);
  }
  // where the granules of 16 keys of this block's range stand in the pools (rows before heads; -1: no query sees one), looked up once
  __shared__ long long granule_s[TT_GRANULES];
  const int g_first = k_first / 16, n_granules = k_first <= k_last ? (k_last - k_first) / TT_BN * (TT_BN / 16) + TT_BN / 16 : 0;
  auto granule = [&](int i) {
    const int p0 = (g_first + i) * 16, blk = p0 / a.page_size;
    return p0 + 15 >= lo0 && p0 <= pos_last ? (long long)table[blk] * G * a.page_size + (p0 - blk * a.page_size) : -1;
  };
  for (int i = tid; i < min(n_granules, TT_GRANULES); i += nthreads) granule_s[i] = granule(i);
  __syncthreads();
  // keys or values of a tile: a thread takes 16-byte pieces (key, column), of every head the same
  auto copy_pieces = [&](int k0, __nv_bfloat16* dst, const __nv_bfloat16* pool, int width, int pieces, int ld) {
    const long long head_step = (long long)a.page_size * width;
    for (int i = tid; i < TT_BN * pieces; i += nthreads) {
      const int j = i / pieces, c = (i - j * pieces) * 8, pj = k0 + j;
      const int at = (pj >> 4) - g_first;
      const long long row = at < TT_GRANULES ? granule_s[at] : granule(at);
      __nv_bfloat16* to = dst + (size_t)j * ld + c;
      if (row >= 0 && pj >= lo0 && pj <= pos_last) {
        const __nv_bfloat16* from = pool + (row + (pj & 15)) * width + c;
        for (int g = 0; g < G; g++, to += (size_t)TT_BN * ld, from += head_step) tt_cp_async16(to, from);
      } else {
        for (int g = 0; g < G; g++, to += (size_t)TT_BN * ld) *reinterpret_cast<uint4*>(to) = make_uint4(0, 0, 0, 0);
      }
    }
    tt_cp_async_commit();
  };
  auto copy = [&](int k0, bool values) {
    if (values) copy_pieces(k0, Vs, a.v_pool, VDIM, VDIM / 8, vs_ld);
    else copy_pieces(k0, Ks, a.k_pool, dim, dv8, qs_ld);
  };
  // The same by tensor copies of 16 keys x 64 channels of a head.  One thread says how many bytes are coming (before the barrier that frees
  // the buffer), then every warp sends for some of them, so that no warp stands long at the unit, which takes 67 cycles a copy.
  // A granule that no query sees is not fetched: its scores are masked, its values cleared.
  auto expect = [&](int k0, bool values) {
    if (tid) return;
    int n = 0;
#pragma unroll
    for (int i = 0; i < TT_BN / 16; i++) n += k0 + 16 * i + 15 >= lo0 && k0 + 16 * i <= pos_last;
    tt_expect(values ? v_full : k_full, (uint32_t)(n * G * 16 * 2 * (values ? VDIM : dim)));
  };
  auto fetch = [&](int k0, bool values) {
    if (lane) return;
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");        // what was read there, before it is written
    const int spans = (values ? VDIM : dim) / 64, per = (TT_BN / 16) * spans;
    for (int i = warp; i < G * per; i += nthreads >> 5) {
      const int g = i / per, gran = (i - g * per) / spans, span = i % spans, at = k0 / 16 + gran - g_first;
      const long long row = at < TT_GRANULES ? granule_s[at] : granule(at);
      if (row < 0) continue;
      tt_tensor_copy(tt_addr(values ? Vs : Ks) + ((g * spans + span) * TT_BN + gran * 16) * 128, values ? &map_v : &map_k, span * 64,
                     (int)row + g * a.page_size, values ? v_full : k_full);
    }
  };
  if (TENSOR) {
    if (k_first <= k_last) expect(k_first, false);
    __syncthreads();
    if (k_first <= k_last) fetch(k_first, false);
  } else if (k_first <= k_last) {
    copy(k_first, false);
  }
  const float cap_scale = a.softcap > 0.f ? a.scale / a.softcap : a.scale;
  for (int k0 = k_first; k0 <= k_last; k0 += TT_BN) {
    const uint32_t parity = (uint32_t)((k0 - k_first) / TT_BN) & 1;
    if (TENSOR) expect(k0, true);
    else tt_cp_async_wait<0>();
    __syncthreads();       // the tile before is done with Vs and sc (and Qs, tk are written); copied rows are there for all
    if (TENSOR) {
      fetch(k0, true);
      tt_wait(k_full, parity, a.status, 91);
    } else {
      copy(k0, true);
    }

    // 1. raw scores of this warp's head
    if (has_head) {
      float s[TT_BN / 8][4];
#pragma unroll
      for (int nt = 0; nt < TT_BN / 8; nt++) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
      // matrices of 8 x 8: of the queries rows 0-7, 8-15 at columns kk, then at kk + 8; of the keys eight keys at
      // columns kk and kk + 8, then the next eight
      const __nv_bfloat16* qh = Qs + ((size_t)warp * TT_BM + (lane & 15)) * qs_ld + (lane >> 4) * 8;
      const __nv_bfloat16* kg = Ks + ((size_t)g_own * TT_BN + (lane >> 4) * 8 + (lane & 7)) * qs_ld + (lane >> 3 & 1) * 8;
      if constexpr (TENSOR) {
        // a piece's place is its number exchanged with the row's: one exclusive or an address
        const uint32_t ka = tt_addr(Ks) + (uint32_t)(g_own * (DIM / 64) * TT_BN + (lane >> 4) * 8 + (lane & 7)) * 128 +
                            (((lane >> 3 & 1) ^ (lane & 7)) << 4);
#pragma unroll
        for (int kk = 0; kk < DIM; kk += 16) {
          uint32_t af[4], bf[4];
          tt_ldmatrix_x4(af, qh + kk);
#pragma unroll
          for (int nt = 0; nt < TT_BN / 8; nt += 2) {
            tt_ldmatrix_x4(bf, (ka ^ ((kk & 63) >> 3 << 4)) + ((kk >> 6) * TT_BN + nt * 8) * 128);
            tt_mma(s[nt], af, bf[0], bf[1]);
            tt_mma(s[nt + 1], af, bf[2], bf[3]);
          }
        }
      } else {
#pragma unroll 4
        for (int kk = 0; kk < dim; kk += 16) {
          uint32_t af[4], bf[4];
          tt_ldmatrix_x4(af, qh + kk);
#pragma unroll
          for (int nt = 0; nt < TT_BN / 8; nt += 2) {
            tt_ldmatrix_x4(bf, kg + (size_t)nt * 8 * qs_ld + kk);
            tt_mma(s[nt], af, bf[0], bf[1]);
            tt_mma(s[nt + 1], af, bf[2], bf[3]);
          }
        }
      }
      float* sh = sc + (size_t)warp * sc_hd;
#pragma unroll
      for (int nt = 0; nt < TT_BN / 8; nt++) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float v = s[nt][e] * cap_scale;
          s[nt][e] = a.softcap > 0.f ? a.softcap * tt_tanh(v) : v;
        }
        *reinterpret_cast<float2*>(sh + (size_t)r0 * sc_ld + nt * 8 + c2) = make_float2(s[nt][0], s[nt][1]);
        *reinterpret_cast<float2*>(sh + (size_t)(r0 + 8) * sc_ld + nt * 8 + c2) = make_float2(s[nt][2], s[nt][3]);
      }
    }
    const bool more = k0 + TT_BN <= k_last;
    if (TENSOR && more) expect(k0 + TT_BN, false);
    __syncthreads();

    // the scores are written and the keys read: the next tile's keys may come
    if (TENSOR) {
      if (more) fetch(k0 + TT_BN, false);
    } else if (more) {
      copy(k0 + TT_BN, false);
    } else {
      tt_cp_async_commit();
    }

    // 2. the heads mixed and the mask: a warp one query and eight keys at a time
    if (a.talk) {
      uint32_t t[3][4];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) t[i][e] = tk[(i * 4 + e) * 32 + lane];
      for (int unit = warp; unit < rows * (TT_BN / 8); unit += nthreads >> 5) {
        const int r = unit / (TT_BN / 8), n0 = (unit - r * (TT_BN / 8)) * 8;
        // B: heads c2, c2 + 1 (and 8 further) of key n0 + r0
        float c[4];
        tt_mix(t, sc + (size_t)r * sc_ld + n0 + r0, sc_hd, H, c2, c);
        const int pi = pos0 + r, pj = k0 + n0 + c2, first = first_s[r];
        const bool ok0 = pj >= first && pj <= pi, ok1 = pj + 1 >= first && pj + 1 <= pi;
        float* to = sc + (size_t)r * sc_ld + n0 + c2;
        if (r0 < H)
          *reinterpret_cast<float2*>(to + (size_t)r0 * sc_hd) = make_float2(ok0 ? c[0] : -INFINITY, ok1 ? c[1] : -INFINITY);
        if (r0 + 8 < H)
          *reinterpret_cast<float2*>(to + (size_t)(r0 + 8) * sc_hd) =
              make_float2(ok0 ? c[2] : -INFINITY, ok1 ? c[3] : -INFINITY);
      }
    } else {
      // no matrix: the mask alone (the identity's zeros would let what is not finite in one head into all of them)
      for (int i = tid; i < H * rows * TT_BN; i += nthreads) {
        const int h = i / (rows * TT_BN), r = (i - h * rows * TT_BN) / TT_BN, key = i % TT_BN, pj = k0 + key;
        if (pj < first_s[r] || pj > pos0 + r) sc[(size_t)h * sc_hd + r * sc_ld + key] = -INFINITY;
      }
    }
    if (TENSOR) {
      tt_wait(v_full, parity, a.status, 92);
      // values of keys that no query of the tile sees are stale memory: a weight of zero times them has to be zero
      if (k0 < lo0 || k0 + TT_BN - 1 > pos_last)
        for (int i = tid; i < G * TT_BN * (VDIM / 8); i += nthreads) {
          const int key = k0 + i / 8 % TT_BN;
          if (key < lo0 || key > pos_last) reinterpret_cast<uint4*>(Vs)[i] = make_uint4(0, 0, 0, 0);
        }
    } else {
      tt_cp_async_wait<1>();      // the values are there; the next keys may still be on their way
    }
    __syncthreads();

    // 3. softmax of the mixed scores and the product with the values
    if (has_head) {
      const float* sh = sc + (size_t)warp * sc_hd;
      float s[TT_BN / 8][4];
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int nt = 0; nt < TT_BN / 8; nt++) {
        float2 x = *reinterpret_cast<const float2*>(sh + (size_t)r0 * sc_ld + nt * 8 + c2);
        float2 y = *reinterpret_cast<const float2*>(sh + (size_t)(r0 + 8) * sc_ld + nt * 8 + c2);
        if (r0 >= rows) x = make_float2(-INFINITY, -INFINITY);          // rows beyond the portion were not mixed
        if (r0 + 8 >= rows) y = make_float2(-INFINITY, -INFINITY);
        s[nt][0] = x.x; s[nt][1] = x.y; s[nt][2] = y.x; s[nt][3] = y.y;
        mx[0] = fmaxf(mx[0], fmaxf(x.x, x.y));
        mx[1] = fmaxf(mx[1], fmaxf(y.x, y.y));
      }
      float alpha[2], m_log2[2];           // maxima in powers of two; 0 while a row has no key
#pragma unroll
      for (int e = 0; e < 2; e++) {
        mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
        mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
        const float m_new = fmaxf(m_run[e], mx[e]);
        m_log2[e] = m_new == -INFINITY ? 0.f : tt_max_log2(m_new);
        alpha[e] = tt_exp2(tt_max_log2(m_run[e]) - m_log2[e]);
        m_run[e] = m_new;
      }
      float sum[2] = {0.f, 0.f};
#pragma unroll
      for (int nt = 0; nt < TT_BN / 8; nt++) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float p = tt_exp2(fmaf(s[nt][e], TT_LOG2E, -m_log2[e >> 1]));        // 0 of -infinity
          s[nt][e] = p;
          sum[e >> 1] += p;
        }
      }
      l_run[0] = l_run[0] * alpha[0] + sum[0];
      l_run[1] = l_run[1] * alpha[1] + sum[1];
      if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
        for (int i = 0; i < VDIM / 8; i++) {
          o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
          o[i][2] *= alpha[1]; o[i][3] *= alpha[1];
        }
      }
      const __nv_bfloat16* vg = Vs + (size_t)g_own * TT_BN * vs_ld;
      const uint32_t va = tt_addr(Vs) + (uint32_t)(g_own * (VDIM / 64) * TT_BN + (lane & 15)) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
#pragma unroll
      for (int ks = 0; ks < TT_BN / 16; ks++) {
        uint32_t pf[4];
        pf[0] = tt_pack(s[2 * ks][0], s[2 * ks][1]);
        pf[1] = tt_pack(s[2 * ks][2], s[2 * ks][3]);
        pf[2] = tt_pack(s[2 * ks + 1][0], s[2 * ks + 1][1]);
        pf[3] = tt_pack(s[2 * ks + 1][2], s[2 * ks + 1][3]);
#pragma unroll
        for (int nt = 0; nt < VDIM / 8; nt += 2) {
          uint32_t bf[4];        // keys 0-7 and 8-15 of the step at eight columns, then at the next eight
          if (TENSOR)
            tt_ldmatrix_x4_trans(bf, (va ^ ((nt & 7) << 4)) + ((nt >> 3) * TT_BN + ks * 16) * 128);
          else
            tt_ldmatrix_x4_trans(bf, vg + (size_t)(ks * 16 + (lane & 15)) * vs_ld + nt * 8 + (lane >> 4) * 8);
          tt_mma(o[nt], pf, bf[0], bf[1]);
          tt_mma(o[nt + 1], pf, bf[2], bf[3]);
        }
      }
    }
  }

  if (has_head) {
#pragma unroll
    for (int e = 0; e < 2; e++) {
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 1);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 2);
    }
    if (a.splits > 0) {      // the split's unnormalised rows with their maximum and sum
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const int r = r0 + 8 * half;
        if (r < rows) {
          const long long slot = ((long long)(q_start + row0 + r) * a.splits + blockIdx.z) * H + warp;
          if (m_run[half] != -INFINITY)      // a split without a key for the row is never read
#pragma unroll
          for (int nt = 0; nt < VDIM / 8; nt++)
            *reinterpret_cast<float2*>(a.part_o + slot * VDIM + nt * 8 + c2) =
                make_float2(o[nt][2 * half], o[nt][2 * half + 1]);
          if (c2 == 0) {
            a.part_ml[slot * 2] = tt_max_log2(m_run[half]);
            a.part_ml[slot * 2 + 1] = l_run[half];
          }
        }
      }
      return;
    }
    const float inv0 = 1.0f / l_run[0], inv1 = 1.0f / l_run[1];
#pragma unroll
    for (int nt = 0; nt < VDIM / 8; nt++) {
      if (r0 < rows)
        *reinterpret_cast<__nv_bfloat162*>(a.out + ((long long)(q_start + row0 + r0) * H + warp) * VDIM + nt * 8 + c2) =
            __floats2bfloat162_rn(o[nt][0] * inv0, o[nt][1] * inv0);
      if (r0 + 8 < rows)
        *reinterpret_cast<__nv_bfloat162*>(a.out + ((long long)(q_start + row0 + r0 + 8) * H + warp) * VDIM + nt * 8 + c2) =
            __floats2bfloat162_rn(o[nt][2] * inv1, o[nt][3] * inv1);
    }
  }
}

static size_t tt_smem_bytes(int H, int G, int dim, int vdim) {
  return (size_t)(H * TT_BM + G * TT_BN) * (dim + 8) * 2 + (size_t)G * TT_BN * (vdim + 8) * 2 +
         (size_t)H * (TT_BM * (TT_BN + TT_SPAD) + 4) * 4 + 3 * 4 * 32 * 4;
}

// 1 if the kernel takes these sizes
MF_API int mf_attention_talking_tc_ok(int n_heads, int n_kv, int dim, int vdim, int page_size) {
  if (n_heads < 1 || n_heads > 16 || n_kv < 1 || n_heads % n_kv) return 0;
  if (dim % 16 || dim < 16 || dim > 256) return 0;
  if (vdim != 32 && vdim != 64 && vdim != 96 && vdim != 128) return 0;
  if (page_size % 16) return 0;
  return tt_smem_bytes(n_heads, n_kv, dim, vdim) <= 200 * 1024 ? 1 : 0;
}

// out[t, h] = sum_z o_z 2^{m_z - m} / sum_z l_z 2^{m_z - m}, the splits in their order; a warp per (token, head), VDIM / 32
// neighbouring channels a lane
template <int VDIM>
__global__ void __launch_bounds__(256)
talking_attention_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                               __nv_bfloat16* __restrict__ out, int splits, int H, int first_row, int n) {
  constexpr int N = VDIM / 32;
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), c = (threadIdx.x & 31) * N;
  if (item >= n) return;
  const int t = first_row + item / H, h = item % H;
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + (long long)t * splits * H + h;
  const float* po = part_o + ((long long)t * splits * H + h) * VDIM + c;
  if (ml[0].y == -1.f) return;          // keys of one cut: their block has written the row
  float m = -INFINITY;
  for (int z = 0; z < splits; z++) m = fmaxf(m, ml[(long long)z * H].x);
  float l = 0.f, acc[N];
#pragma unroll
  for (int i = 0; i < N; i++) acc[i] = 0.f;
  for (int z = 0; z < splits; z++) {
    const float2 x = ml[(long long)z * H];
    const bool none = x.x == -INFINITY;           // no key, a sum of 0; or no key whose score is a number, and then it is none
    const float w = none ? 1.f : tt_exp2(x.x - m);
    l = fmaf(x.y, w, l);
    if (none) continue;
#pragma unroll
    for (int i = 0; i < N; i++) acc[i] += po[(long long)z * H * VDIM + i] * w;
  }
  const float inv = 1.0f / l;
#pragma unroll
  for (int i = 0; i < N; i++) out[((long long)t * H + h) * VDIM + c + i] = __float2bfloat16_rn(acc[i] * inv);
}

// One query per sequence: a block per (sequence, split of TT_SPAN keys), eight warps.  Here the rows of a product are the query heads
// of one key head, not queries (the kernel above has one of 16 rows filled): S = Q K^T by units of a key head and 16 keys with the
// keys read straight into the operand's registers (both factors take the channels of a step of 16 in the same other order, so a
// thread reads 8 neighbouring bytes), the heads mixed as above, one softmax over the split, O = P V by units of a key head and 16
// channels.  The values come by cp.async from the start.  Bound by memory latency where the splits are few and by the bandwidth where
// they are many:
// the layer's step, 16 / 4 heads of 128, 8 sequences of 2,000 keys 78.9 -> 33.2 us with the merge below against the kernel above
// over splits of 128 keys, one sequence 69.7 -> 22.6, 32 sequences of 8 / 2 heads 60.0 -> 28.8.
#define TT_SPAN (TT_SPLIT_TILES * TT_BN)
static size_t tt_decode_smem(int H, int G, int vdim) {
  return (size_t)G * TT_SPAN * (vdim + 8) * 2 + (size_t)H * (TT_SPAN + 4) * 4 + (size_t)H * (TT_SPAN + 8) * 2;
}

template <int VDIM>
__global__ void __launch_bounds__(256, 2)
talking_decode_kernel(const TtArgs a) {
  extern __shared__ __align__(16) unsigned char tt_smem[];
  __shared__ uint32_t tk[3 * 4 * 32];
  const int H = a.n_heads, G = a.n_kv, dim = a.dim, rep = H / G;
  constexpr int vs_ld = VDIM + 8, sc_ld = TT_SPAN + 4, p_ld = TT_SPAN + 8, STEPS = 8;
  __nv_bfloat16* Vs = reinterpret_cast<__nv_bfloat16*>(tt_smem);             // [G][TT_SPAN][vs_ld]
  float* sc = reinterpret_cast<float*>(Vs + (size_t)G * TT_SPAN * vs_ld);    // [H][sc_ld]
  __nv_bfloat16* Ps = reinterpret_cast<__nv_bfloat16*>(sc + H * sc_ld);      // [H][p_ld]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = lane >> 2, c2 = (lane & 3) * 2;
  pdl_launch();
  if (warp < 4) tt_talk_pieces(a.talk, H, warp, lane, tk);
  pdl_wait();

  const int seq = blockIdx.y, split = blockIdx.x;
  const int pos = a.seq_ctx_len[seq] - 1, row = a.seq_q_start[seq];
  const int* table = a.block_table + (long long)(a.table_row0 + seq) * a.bt_stride;
  int first = 0;
  if (a.window > 0) first = max(first, pos - a.window + 1);
  if (a.chunk > 0) first = max(first, pos / a.chunk * a.chunk);
  const int k0 = (first / TT_SPAN + split) * TT_SPAN;
  const int k_lo = max(first, k0), k_hi = min(pos, k0 + TT_SPAN - 1);
  const long long slot0 = ((long long)row * a.splits + split) * H;
  if (k_lo > k_hi) {
    if (tid < H) {
      a.part_ml[(slot0 + tid) * 2] = -INFINITY;
      a.part_ml[(slot0 + tid) * 2 + 1] = 0.f;
    }
    return;
  }
  for (int i = tid; i < TT_SPAN * (VDIM / 8); i += 256) {
    const int j = i / (VDIM / 8), c = (i - j * (VDIM / 8)) * 8, pj = k0 + j, blk = pj / a.page_size;
    const bool in = pj >= k_lo && pj <= k_hi;
    const __nv_bfloat16* from =
        a.v_pool + ((in ? (long long)table[blk] : 0) * G * a.page_size + (pj - blk * a.page_size)) * VDIM + c;
    __nv_bfloat16* to = Vs + (size_t)j * vs_ld + c;
    for (int g = 0; g < G; g++, to += (size_t)TT_SPAN * vs_ld, from += (long long)a.page_size * VDIM) {
      if (in) tt_cp_async16(to, from);
      else *reinterpret_cast<uint4*>(to) = make_uint4(0, 0, 0, 0);
    }
  }
  tt_cp_async_commit();

  // scores: 16 keys lie in one page; keys of them that the query does not see only make scores that the mask drops
  const float cap_scale = a.softcap > 0.f ? a.scale / a.softcap : a.scale;
  for (int u = warp; u < G * (TT_SPAN / 16); u += 8) {
    const int g = u / (TT_SPAN / 16), j = (u - g * (TT_SPAN / 16)) * 16;
    if (k0 + j > k_hi || k0 + j + 15 < k_lo) continue;
    const int blk = (k0 + j) / a.page_size;
    const __nv_bfloat16* kp = a.k_pool + (((long long)table[blk] * G + g) * a.page_size + (k0 + j - blk * a.page_size) + r0) * dim +
                              2 * c2;
    const __nv_bfloat16* qp = a.q + ((long long)row * H + g * rep + r0) * dim + 2 * c2;
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    for (int kk = 0; kk < dim; kk += 16 * STEPS) {
      uint2 kf[STEPS][2], qf[STEPS][2];
#pragma unroll
      for (int i = 0; i < STEPS; i++) {
        const int c = kk + i * 16;
        const bool in = c < dim;
        const uint2 zero = make_uint2(0, 0);
        kf[i][0] = in ? *reinterpret_cast<const uint2*>(kp + c) : zero;
        kf[i][1] = in ? *reinterpret_cast<const uint2*>(kp + 8 * dim + c) : zero;
        qf[i][0] = in && r0 < rep ? *reinterpret_cast<const uint2*>(qp + c) : zero;
        qf[i][1] = in && r0 + 8 < rep ? *reinterpret_cast<const uint2*>(qp + 8 * dim + c) : zero;
      }
#pragma unroll
      for (int i = 0; i < STEPS; i++) {
        const uint32_t af[4] = {qf[i][0].x, qf[i][1].x, qf[i][0].y, qf[i][1].y};
        tt_mma(s[0], af, kf[i][0].x, kf[i][0].y);
        tt_mma(s[1], af, kf[i][1].x, kf[i][1].y);
      }
    }
    float* to = sc + (size_t)(g * rep + r0) * sc_ld + j + c2;
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float v = s[nt][e] * cap_scale;
        s[nt][e] = a.softcap > 0.f ? a.softcap * tt_tanh(v) : v;
      }
      if (r0 < rep) *reinterpret_cast<float2*>(to + nt * 8) = make_float2(s[nt][0], s[nt][1]);
      if (r0 + 8 < rep) *reinterpret_cast<float2*>(to + 8 * sc_ld + nt * 8) = make_float2(s[nt][2], s[nt][3]);
    }
  }
  __syncthreads();

  // the heads mixed, eight keys a warp; a key's scores meet no other key's
  for (int n0 = warp * 8; n0 < TT_SPAN; n0 += 64) {
    uint32_t t[3][4];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int e = 0; e < 4; e++) t[i][e] = tk[(i * 4 + e) * 32 + lane];
    float c[4];
    if (a.talk) {
      tt_mix(t, sc + n0 + r0, sc_ld, H, c2, c);
    } else {                     // no matrix: a head's own scores (the identity's zeros would let what is not finite into all heads)
#pragma unroll
      for (int e = 0; e < 4; e++) c[e] = r0 + (e & 2) * 4 < H ? sc[(r0 + (e & 2) * 4) * sc_ld + n0 + c2 + (e & 1)] : 0.f;
    }
    const int pj = k0 + n0 + c2;
    const bool ok0 = pj >= k_lo && pj <= k_hi, ok1 = pj + 1 >= k_lo && pj + 1 <= k_hi;
    float* to = sc + n0 + c2;
    __syncwarp();
    if (r0 < H) *reinterpret_cast<float2*>(to + r0 * sc_ld) = make_float2(ok0 ? c[0] : -INFINITY, ok1 ? c[1] : -INFINITY);
    if (r0 + 8 < H)
      *reinterpret_cast<float2*>(to + (r0 + 8) * sc_ld) = make_float2(ok0 ? c[2] : -INFINITY, ok1 ? c[3] : -INFINITY);
  }
  __syncthreads();

  // softmax of the split, a warp a head
  for (int h = warp; h < H; h += 8) {
    const float2 x = *reinterpret_cast<const float2*>(sc + h * sc_ld + lane * 2);
    float m = fmaxf(x.x, x.y);
#pragma unroll
    for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    const float m_log2 = m == -INFINITY ? 0.f : tt_max_log2(m);
    const float p0 = tt_exp2(fmaf(x.x, TT_LOG2E, -m_log2)), p1 = tt_exp2(fmaf(x.y, TT_LOG2E, -m_log2));
    const float l = warp_sum(p0 + p1);
    *reinterpret_cast<uint32_t*>(Ps + h * p_ld + lane * 2) = tt_pack(p0, p1);
    if (lane == 0) {
      a.part_ml[(slot0 + h) * 2] = tt_max_log2(m);
      a.part_ml[(slot0 + h) * 2 + 1] = l;
    }
  }
  tt_cp_async_wait<0>();
  __syncthreads();

  for (int u = warp; u < G * (VDIM / 16); u += 8) {
    const int g = u / (VDIM / 16), n = (u - g * (VDIM / 16)) * 16;
    const __nv_bfloat16* p = Ps + (size_t)(g * rep + r0) * p_ld + c2;
    const __nv_bfloat16* v = Vs + ((size_t)g * TT_SPAN + (lane & 15)) * vs_ld + n + (lane >> 4) * 8;
    float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < TT_SPAN; ks += 16) {
      uint32_t pf[4] = {0, 0, 0, 0}, bf[4];
      if (r0 < rep) {
        pf[0] = *reinterpret_cast<const uint32_t*>(p + ks);
        pf[2] = *reinterpret_cast<const uint32_t*>(p + ks + 8);
      }
      if (r0 + 8 < rep) {
        pf[1] = *reinterpret_cast<const uint32_t*>(p + 8 * p_ld + ks);
        pf[3] = *reinterpret_cast<const uint32_t*>(p + 8 * p_ld + ks + 8);
      }
      tt_ldmatrix_x4_trans(bf, v + (size_t)ks * vs_ld);
      tt_mma(o[0], pf, bf[0], bf[1]);
      tt_mma(o[1], pf, bf[2], bf[3]);
    }
    float* to = a.part_o + (slot0 + g * rep + r0) * VDIM + n + c2;
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      if (r0 < rep) *reinterpret_cast<float2*>(to + nt * 8) = make_float2(o[nt][0], o[nt][1]);
      if (r0 + 8 < rep) *reinterpret_cast<float2*>(to + 8 * VDIM + nt * 8) = make_float2(o[nt][2], o[nt][3]);
    }
  }
}

// The merge of a decode step, whose rows are few and whose splits many: a block per (token, head), eight warps that take every
// eighth split each.
template <int VDIM>
__global__ void __launch_bounds__(256)
talking_decode_merge_kernel(const float* part_o, const float* part_ml, __nv_bfloat16* __restrict__ out,
                            int splits, int H) {
  constexpr int N = VDIM / 32;
  __shared__ float m_s[8], l_s[8], o_s[8][VDIM];
  const int t = blockIdx.x / H, h = blockIdx.x - t * H, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_launch();
  pdl_wait();
  const float2* ml = reinterpret_cast<const float2*>(part_ml) + (long long)t * splits * H + h;
  const float* po = part_o + ((long long)t * splits * H + h) * VDIM + lane;
  float m = -INFINITY;
  for (int z = threadIdx.x; z < splits; z += 256) m = fmaxf(m, ml[(long long)z * H].x);
#pragma unroll
  for (int off = 16; off; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if (lane == 0) m_s[warp] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; w++) m = fmaxf(m, m_s[w]);
  float l = 0.f, acc[N];
#pragma unroll
  for (int i = 0; i < N; i++) acc[i] = 0.f;
#pragma unroll 4
  for (int z = warp; z < splits; z += 8) {
    const float2 x = ml[(long long)z * H];
    const bool some = x.x != -INFINITY;                       // a split without a key has no output
    const float w = some ? tt_exp2(x.x - m) : 0.f;
    l += x.y * w;
#pragma unroll
    for (int i = 0; i < N; i++) acc[i] += (some ? po[(long long)z * H * VDIM + i * 32] : 0.f) * w;
  }
  if (lane == 0) l_s[warp] = l;
#pragma unroll
  for (int i = 0; i < N; i++) o_s[warp][i * 32 + lane] = acc[i];
  __syncthreads();
  if (threadIdx.x < VDIM) {
    float o = 0.f;
    l = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      o += o_s[w][threadIdx.x];
      l += l_s[w];
    }
    out[(long long)blockIdx.x * VDIM + threadIdx.x] = __float2bfloat16_rn(o * (1.0f / l));
  }
}

template <int VDIM>
static int tt_decode(const TtArgs& a, int n_seqs, cudaStream_t stream) {
  const size_t smem = tt_decode_smem(a.n_heads, a.n_kv, VDIM);
  static DeviceOnce once;
  const int d = mf_current_device();
  if (d < 0) return MF_ERR_BAD_ARG;
  if (!once.done[d]) {
    cudaError_t e = cudaFuncSetAttribute(talking_decode_kernel<VDIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    once.done[d] = true;
  }
  mf_count(MF_K_ATTN_TALKING_DECODE);
  int rc = (int)launch_dep(talking_decode_kernel<VDIM>, dim3(a.splits, n_seqs), dim3(256), smem, stream, a);
  if (rc != 0) return rc;
  mf_count(MF_K_ATTN_TALKING_MERGE);
  return (int)launch_dep(talking_decode_merge_kernel<VDIM>, dim3(n_seqs * a.n_heads), dim3(256), 0, stream, (const float*)a.part_o,
                         (const float*)a.part_ml, a.out, a.splits, a.n_heads);
}

static int tt_merge(const float* part_o, const float* part_ml, void* out, int splits, int H, int vdim, int first_row,
                    int n_rows, cudaStream_t stream) {
  const int n = n_rows * H;
  mf_count(MF_K_ATTN_TALKING_MERGE);
#define TT_MERGE(VD)                                                                                                       \
  if (vdim == VD)                                                                                                          \
  talking_attention_merge_kernel<VD><<<(n + 7) / 8, 256, 0, stream>>>(part_o, part_ml, (__nv_bfloat16*)out, splits, H, first_row, n)
  TT_MERGE(32);
  TT_MERGE(64);
  TT_MERGE(96);
  TT_MERGE(128);
#undef TT_MERGE
  return (int)cudaGetLastError();
}

// Key tiles of a split for portions of prompts: by the lane's mask alone, so that the order of a row's sums is its own.
static int tt_prefill_split_tiles(int window, int chunk) {
  const int most = window > 0 && chunk > 0 ? (window < chunk ? window : chunk) : (window > 0 ? window : chunk);
  return most > 0 && most <= 4096 ? TT_PREFILL_SPLIT_TILES / 2 : TT_PREFILL_SPLIT_TILES;
}

template <int VDIM, int MAXH, int DIM>
static int tt_launch_as(const CUtensorMap& mk, const CUtensorMap& mv, const TtArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
  const size_t smem = tt_smem_bytes(a.n_heads, a.n_kv, a.dim, VDIM);
  static DeviceOnce once;
  const int d = mf_current_device();
  if (d < 0) return MF_ERR_BAD_ARG;
  if (!once.done[d]) {
    cudaError_t e = cudaFuncSetAttribute(talking_attention_tc_kernel<VDIM, MAXH, DIM>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    once.done[d] = true;
  }
  mf_count(MF_K_ATTN_TALKING_MMA);
  dim3 grid((max_q_len + TT_BM - 1) / TT_BM, n_seqs, a.splits > 0 ? a.splits : 1);
  const int warps = a.n_heads < 4 ? 4 : a.n_heads;       // at least four warps for the loads and the mixing
  talking_attention_tc_kernel<VDIM, MAXH, DIM><<<grid, 32 * warps, smem, stream>>>(mk, mv, a);
  return (int)cudaGetLastError();
}

template <int VDIM, int MAXH>
static int tt_launch(const TtArgs& a, int n_seqs, int max_q_len, cudaStream_t stream) {
  CUtensorMap mk = {}, mv = {};
  if constexpr (VDIM % 64 == 0) {
    if ((a.dim == 64 || a.dim == 128) && a.pool_rows > 0 && !(((uintptr_t)a.k_pool | (uintptr_t)a.v_pool) & 15)) {
      int rc = tma_host::bf16_map(a.k_pool, a.pool_rows, a.dim, 16, 64, &mk);
      if (rc == 0) rc = tma_host::bf16_map(a.v_pool, a.pool_rows, VDIM, 16, 64, &mv);
      if (rc) return rc;
      if (a.dim == 64) return tt_launch_as<VDIM, MAXH, 64>(mk, mv, a, n_seqs, max_q_len, stream);
      return tt_launch_as<VDIM, MAXH, 128>(mk, mv, a, n_seqs, max_q_len, stream);
    }
  }
  return tt_launch_as<VDIM, MAXH, 0>(mk, mv, a, n_seqs, max_q_len, stream);
}

// The sequences described by the three per-sequence arrays start at row `table_row0` of the
// block table; q and out are the whole step's [T, n_heads * dim] and [T, n_heads * vdim].
MF_API int mf_attention_talking_tc(const void* q, const void* k_pool, const void* v_pool, void* out,
                                   const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len,
                                   int table_row0, int n_seqs, int max_q_len, int n_heads, int n_kv, int dim, int vdim,
                                   const int* block_table, int bt_stride, int page_size, long long pool_rows, float scale, float softcap,
                                   const float* talk, int window, int chunk, int splits, float* part_o, float* part_ml,
                                   int first_row, int n_rows, int min_ctx, int max_ctx, int* status,
                                   cudaStream_t stream) {
  if (n_seqs <= 0 || max_q_len <= 0) return 0;
  if (!mf_attention_talking_tc_ok(n_heads, n_kv, dim, vdim, page_size) || n_seqs > 65535 || splits < 0 || splits > 65535)
    return MF_ERR_BAD_ARG;
  TtArgs a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, (__nv_bfloat16*)out,
           seq_q_start, seq_q_len, seq_ctx_len, block_table, talk, table_row0, bt_stride, page_size, n_heads, n_kv, dim,
           scale, softcap, window, chunk, splits, tt_prefill_split_tiles(window, chunk), part_o, part_ml, status, pool_rows, 0};
  mf_count(MF_K_ATTN_TALKING_TC);
  int rc = MF_ERR_BAD_ARG;
  // A sequence goes to either kernel by its own length, so that its numbers do not depend on what else is in the step; a kernel that no
  // sequence goes to is not launched.
  const int from = talking_prompt_from(n_heads), least = talking_prompt_keys(min_ctx, window, chunk),
            most = talking_prompt_keys(max_ctx > 0 ? max_ctx : 1 << 30, window, chunk);
  const bool takes = most >= from && talking_prompt_takes(n_heads, n_kv, dim, vdim, q, k_pool, v_pool, pool_rows);
  if (takes) {
    const int cuts = talking_prompt_cuts(splits, chunk);
    mf_count(MF_K_ATTN_TALKING_PROMPT);
    rc = talking_prompt_launch(q, k_pool, v_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs, max_q_len, n_heads,
                               block_table, bt_stride, page_size, pool_rows, scale, softcap, talk, window, chunk, cuts,
                               from, part_o, part_ml, status, stream);
    mf_count_own(cuts > 1 ? 2 : 1);
    if (rc == 0 && cuts > 1) rc = tt_merge(part_o, part_ml, out, cuts, n_heads, vdim, first_row, n_rows, stream);
    if (rc != 0 || least >= from) return rc;
    a.below_keys = from, a.splits = splits = 0;          // of the short ones a block walks all keys
  }
#define TT_CASE(VD)                                                         \
  if (vdim == VD)                                                           \
    rc = n_heads <= 8 ? tt_launch<VD, 8>(a, n_seqs, max_q_len, stream) : tt_launch<VD, 16>(a, n_seqs, max_q_len, stream);
  TT_CASE(32)
  TT_CASE(64)
  TT_CASE(96)
  TT_CASE(128)
#undef TT_CASE
  mf_count_own(splits > 0 ? 2 : 1);
  if (rc != 0 || splits == 0) return rc;
  // the rows of the portions are rows first_row .. first_row + n_rows of the step
  return tt_merge(part_o, part_ml, out, splits, n_heads, vdim, first_row, n_rows, stream);
}

// Splits of a launch for portions of prompts whose queries see at most `max_keys` keys (0: none needed).
MF_API int mf_attention_talking_prefill_splits(int max_keys, int window, int chunk) {
  const int tiles = (max_keys + TT_BN - 1) / TT_BN + 1, per = tt_prefill_split_tiles(window, chunk);
  if (tiles <= per + 1) return 0;
  return (tiles + per - 1) / per + 1;
}

// Splits that a decode launch needs when no query sees more than `max_keys` keys.
MF_API int mf_attention_talking_splits(int max_keys) {
  const int tiles = (max_keys + TT_BN - 1) / TT_BN + 1;       // a range of keys may straddle one tile more
  return (tiles + TT_SPLIT_TILES - 1) / TT_SPLIT_TILES + 1;   // and one split more
}

// One query per sequence (the newest token of each), keys cut into splits; q and out hold the
// n_seqs tokens, row t the token of row t of the block table.  part_o needs
// n_seqs * splits * n_heads * vdim floats, part_ml n_seqs * splits * n_heads * 2.
MF_API int mf_attention_talking_decode(const void* q, const void* k_pool, const void* v_pool, void* out,
                                       const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len, int n_seqs,
                                       int n_heads, int n_kv, int dim, int vdim, const int* block_table, int bt_stride,
                                       int page_size, long long pool_rows, float scale, float softcap, const float* talk, int window,
                                       int chunk, int splits, float* part_o, float* part_ml, int* status, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (!mf_attention_talking_tc_ok(n_heads, n_kv, dim, vdim, page_size) || n_seqs > 65535 || splits < 1 || splits > 65535)
    return MF_ERR_BAD_ARG;
  TtArgs a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, (__nv_bfloat16*)out,
           seq_q_start, seq_q_len, seq_ctx_len, block_table, talk, 0, bt_stride, page_size, n_heads, n_kv, dim,
           scale, softcap, window, chunk, splits, TT_SPLIT_TILES, part_o, part_ml, status, pool_rows, 0};
  mf_count(MF_K_ATTN_TALKING_TC);
  // the values of all key heads of a split have to fit in shared memory; what is wider takes the kernel of the prompts
  if (tt_decode_smem(n_heads, n_kv, vdim) <= 200 * 1024) {
    if (vdim == 32) return tt_decode<32>(a, n_seqs, stream);
    if (vdim == 64) return tt_decode<64>(a, n_seqs, stream);
    if (vdim == 96) return tt_decode<96>(a, n_seqs, stream);
    return tt_decode<128>(a, n_seqs, stream);
  }
  int rc = MF_ERR_BAD_ARG;
#define TT_CASE(VD)                                                         \
  if (vdim == VD) rc = n_heads <= 8 ? tt_launch<VD, 8>(a, n_seqs, 1, stream) : tt_launch<VD, 16>(a, n_seqs, 1, stream);
  TT_CASE(32)
  TT_CASE(64)
  TT_CASE(96)
  TT_CASE(128)
#undef TT_CASE
  if (rc != 0) return rc;
  return tt_merge(part_o, part_ml, out, splits, n_heads, vdim, 0, n_seqs, stream);
}
