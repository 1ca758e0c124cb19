// Paged causal attention of prompt portions for head sizes 64 and 128 on the 5th-generation
// tensor cores: both products of a tile of 128 queries x 64 keys are tcgen05.mma instructions
// with their results in tensor memory, the keys and values come in by TMA, and four warps do
// nothing but the softmax.
//
// A block takes 128 consecutive queries of one head of one sequence and walks the tiles of 64
// keys its queries can see, lowest first, each by the same hand-overs:
//   producer   tensor copies of granules of 16 keys (a page holds whole granules) and 64-wide
//              spans of the head, 128-byte swizzled, into a ring of stages; the queries' own
//              tile once at the start;
//   issuer     one thread: S = Q K^T (M 128, steps of K 16 over the head) into tensor memory,
//              then, when the softmax warps have handed over P, O += P V (V is the N-major
//              operand: its rows are keys, its 128-byte lines run along the head);
//   softmax    a query row per thread (a lane of tensor memory): read the row of S once into
//              registers, mask it where the tile touches the diagonal or a window's end, running
//              maximum and sum in float32, rescale the row of O in tensor memory when the
//              exponent's reference moves (rarely: see MAX_SLACK_LOG2), write the row of P as
//              bfloat16 in the operand layout, at the end divide and store.
// Three kernels: head size 64 (products two tiles ahead of the softmax, two blocks per SM); head
// size 128 and latents (two chains a block); latents whose values are wider than 192 channels
// (products ahead, one block per SM).  Keys outside every query's range in a tile
// may be stale memory: their scores are masked by selection, and their value rows are cleared
// in shared memory before the second product (0 x NaN would poison it).
//
// Every wait is bounded (codes 41-50 in `status`), and the tensor memory is freed in every
// case.  Formula: src/model/sdpa.cpp:71-95; the reference calls its library's fused kernel.
#include "common.cuh"
#include "tma_host.cuh"

namespace {

constexpr int BM = 128;
constexpr int BOX_BYTES = 16 * 64 * 2;             // one tensor copy: 16 keys x 64 values
constexpr int TMEM_COLS = 256;                     // of the kernel for head size 64
constexpr unsigned WAIT_LIMIT = 1u << 26;
constexpr float LOG2E = 1.4426950408889634f;
// The exponent's reference for a row is its running maximum, but it need not be THE maximum:
// any reference cancels in O / l.  A warp moves its rows' references (and rescales its rows of
// O in tensor memory, a load, 64 multiplications and a store per row) only when some row's
// maximum has grown by more than 2^8 since the last move; until then probabilities may reach
// 256, which float32 sums and bfloat16's eight exponent bits hold as well as values below one.
constexpr float MAX_SLACK_LOG2 = 8.0f;
// With options and over a latent the reference IS the maximum: the largest probability of a row is then a 1 that bfloat16
// holds exactly, as in the mma.sync kernel that had these forms before, and the error against 64 bits is the same (a windowed
// layer 0.00369 of the result; 0.00379 with the slack, which took 49 instead of 53 us at 2,237 tokens with one chain a block).
constexpr float EXACT_MAX_LOG2 = 0.0f;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int* status, int code) {
  for (unsigned i = 0; i < WAIT_LIMIT; i++) {
    unsigned done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
  }
  if (status) atomicExch(status, code);
  return false;
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int c0, int c1, int c2, unsigned bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int c0, int c1, unsigned bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// Operand tiles in shared memory are lines of 128 bytes with the 128-byte swizzle, eight lines
// (1024 bytes) to a group.  K-major (Q, K, P): a line is 64 values along the contraction.
// N-major (V): a line is 64 values along N, successive lines are successive contraction
// indices.  Either way groups of eight lines are 1024 bytes apart.
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr >> 4) & 0x3FFF);          // start address
  d |= (unsigned long long)1 << 16;                          // leading byte offset (one 64-wide span: unused)
  d |= (unsigned long long)(1024 >> 4) << 32;                // stride byte offset: 8 lines x 128 B
  d |= (unsigned long long)1 << 46;                          // descriptor version of this architecture
  d |= (unsigned long long)2 << 61;                          // 128-byte swizzle
  return d;
}
__device__ __forceinline__ void umma(unsigned tmem_c, unsigned long long da, unsigned long long db, unsigned idesc,
                                     unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with A in tensor memory: lane = row, two neighbouring k a column
__device__ __forceinline__ void umma_ta(unsigned tmem_c, unsigned tmem_a, unsigned long long db, unsigned idesc,
                                        unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
      ::"r"(tmem_c), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&r)[32]) {
  unsigned u[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]),
        "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
        "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) r[i] = __uint_as_float(u[i]);
}
// The same load in two halves, so that a row's next 32 columns are on their way while the
// current 32 are worked on: `issue` starts it, `landed` waits for every load issued so far.
// `landed` names the registers as operands so that no use of them moves above the wait.
__device__ __forceinline__ void tmem_ld32_issue(unsigned taddr, unsigned (&u)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]),
        "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]),
        "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld32_landed(unsigned (&u)[32]) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;\n"
      : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]),
        "+r"(u[8]), "+r"(u[9]), "+r"(u[10]), "+r"(u[11]), "+r"(u[12]), "+r"(u[13]), "+r"(u[14]), "+r"(u[15]),
        "+r"(u[16]), "+r"(u[17]), "+r"(u[18]), "+r"(u[19]), "+r"(u[20]), "+r"(u[21]), "+r"(u[22]), "+r"(u[23]),
        "+r"(u[24]), "+r"(u[25]), "+r"(u[26]), "+r"(u[27]), "+r"(u[28]), "+r"(u[29]), "+r"(u[30]), "+r"(u[31])
      :: "memory");
}
__device__ __forceinline__ void tmem_st32_issue(unsigned taddr, const float (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      ::"r"(taddr),
        "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])), "r"(__float_as_uint(r[3])),
        "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])), "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])),
        "r"(__float_as_uint(r[8])), "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
        "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])), "r"(__float_as_uint(r[15])),
        "r"(__float_as_uint(r[16])), "r"(__float_as_uint(r[17])), "r"(__float_as_uint(r[18])), "r"(__float_as_uint(r[19])),
        "r"(__float_as_uint(r[20])), "r"(__float_as_uint(r[21])), "r"(__float_as_uint(r[22])), "r"(__float_as_uint(r[23])),
        "r"(__float_as_uint(r[24])), "r"(__float_as_uint(r[25])), "r"(__float_as_uint(r[26])), "r"(__float_as_uint(r[27])),
        "r"(__float_as_uint(r[28])), "r"(__float_as_uint(r[29])), "r"(__float_as_uint(r[30])), "r"(__float_as_uint(r[31]))
      : "memory");
}
__device__ __forceinline__ void tmem_st32(unsigned taddr, const float (&r)[32]) {
  tmem_st32_issue(taddr, r);
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ void sts128(unsigned addr, unsigned a, unsigned b, unsigned c, unsigned d) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// A thread's row of S for 64 keys: read from tensor memory ONCE into `u` (both loads on their
// way before the first is waited for), masked in place where the tile touches the diagonal or a
// window's end (all other tiles take the form without the mask: four integer instructions per
// score less), and its maximum returned.  The second pass works on the registers.
// Keys below `keep` stay visible beside a window.
template <bool EDGE>
__device__ __forceinline__ float row_scores_max(unsigned taddr, unsigned (&u)[2][32], int key0, int my_pos, int my_lo,
                                                int keep = 0) {
  tmem_ld32_issue(taddr, u[0]);
  tmem_ld32_issue(taddr + 32u, u[1]);
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};       // four chains instead of one
#pragma unroll
  for (int c = 0; c < 2; c++) {
    tmem_ld32_landed(u[c]);                      // waits for both; the second call finds them there
    if (EDGE) {
#pragma unroll
      for (int j = 0; j < 32; j++) {
        const int key = key0 + c * 32 + j;
        if (key > my_pos || (key < my_lo && key >= keep)) u[c][j] = __float_as_uint(-INFINITY);
      }
    }
#pragma unroll
    for (int j = 0; j < 32; j += 2)
      mx4[(j >> 1) & 3] = fmax3(mx4[(j >> 1) & 3], __uint_as_float(u[c][j]), __uint_as_float(u[c][j + 1]));
  }
  return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}

// Second pass: probabilities (in place), their sum, and the row of P as bfloat16 in the operand
// layout: 64 keys = the eight 16-byte pieces of the row's 128-byte line.
__device__ __forceinline__ float row_probabilities(unsigned (&u)[2][32], unsigned p_row, int r, float scale_log2,
                                                   float m_off) {
  float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < 2; c++) {
    float (&v)[32] = reinterpret_cast<float (&)[32]>(u[c]);
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const float p = ex2(fmaf(v[j], scale_log2, -m_off));
      v[j] = p;
      sum4[j & 3] += p;
    }
#pragma unroll
    for (int q4 = 0; q4 < 4; q4++) {
      const int piece = c * 4 + q4;
      sts128(p_row + ((piece ^ (r & 7)) << 4), pack_bf16(v[q4 * 8 + 0], v[q4 * 8 + 1]),
             pack_bf16(v[q4 * 8 + 2], v[q4 * 8 + 3]), pack_bf16(v[q4 * 8 + 4], v[q4 * 8 + 5]),
             pack_bf16(v[q4 * 8 + 6], v[q4 * 8 + 7]));
    }
  }
  return (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
}

// The same with P in tensor memory, 32 columns of two keys each.
__device__ __forceinline__ float row_probabilities_tmem(unsigned (&u)[2][32], unsigned tmem_p, float scale_log2, float m_off) {
  float sum4[4] = {0.f, 0.f, 0.f, 0.f};
  float packed[32];
#pragma unroll
  for (int c = 0; c < 2; c++) {
    const float (&v)[32] = reinterpret_cast<const float (&)[32]>(u[c]);
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float p = ex2(fmaf(v[j], scale_log2, -m_off)), q = ex2(fmaf(v[j + 1], scale_log2, -m_off));
      sum4[j & 3] += p;
      sum4[(j & 3) + 1] += q;
      packed[c * 16 + j / 2] = __uint_as_float(pack_bf16(p, q));
    }
  }
  tmem_st32(tmem_p, packed);
  return (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
}

int g_prefill_tc = 1;       // 0: the mma.sync kernel for every shape (mf_set_prefill_tcgen05)

// Options of the kernel with two chains (EX): kept first keys, whose tiles come before the window's; a sink, the running maximum
// and sum a row starts from; a gate on the output row in the epilogue.
struct TcOptions {
  int keep_first;
  const float* sink;
  const __nv_bfloat16* gate;
  long long gate_ld;
  int min_len;              // only portions of at least so many tokens
};
// eight results of a row times sigmoid of eight gates (16-byte aligned)
__device__ __forceinline__ void apply_gate(float* v, const __nv_bfloat16* g) {
  const uint4 u = *reinterpret_cast<const uint4*>(g);
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[2 * i] *= 1.0f / (1.0f + __expf(-__uint_as_float(w[i] << 16)));
    v[2 * i + 1] *= 1.0f / (1.0f + __expf(-__uint_as_float(w[i] & 0xffff0000u)));
  }
}

// ---------------------------------------------------------------------------------------------
// Head size 64 with the products running AHEAD of the softmax.  With one S in tensor memory
// S = Q K^T, the softmax and O += P V of a block would take turns.  Here a block works on sub-tiles of 64 keys and has two
// S buffers (tensor memory: S0 64 columns, S1 64, O 64): while the softmax warps work on
// sub-tile j, S of sub-tile j + 1 is already there and that of j + 2 is issued as soon as P of
// j has been handed over, right behind O += P_j V_j.  The softmax warps never wait for a
// product in the steady state.  Keys and values come in stages of 64 keys (8 KB each, four
// tensor copies of 16 keys) through a ring of five, so that the keys two sub-tiles ahead are
// there when their product is issued.  P stays single: a softmax pass writes it only after
// it has waited for the previous O += P V (which it needs anyway before it rescales O).
namespace ahead {
constexpr int HD = 64, SUB = 64, RING = 5;
constexpr int Q_BYTES = BM * HD * 2, K_BYTES = SUB * HD * 2, STAGE_BYTES = 2 * K_BYTES, P_BYTES = BM * SUB * 2;
constexpr size_t SMEM = Q_BYTES + RING * STAGE_BYTES + P_BYTES + 16 * 8 + 16;
}  // namespace ahead

__global__ void __launch_bounds__(192, 2)
attn_prefill_tc_ahead_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                             const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                             const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                             const int* __restrict__ seq_ctx_len, int table_row0, PagedView pv, int n_heads,
                             float scale_log2, int window, int* __restrict__ status) {
  using namespace ahead;
  extern __shared__ __align__(1024) unsigned char smem[];
  const unsigned q_u = smem_u32(smem), kv_u = q_u + Q_BYTES, p_u = kv_u + RING * STAGE_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + Q_BYTES + RING * STAGE_BYTES + P_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 16);
  const unsigned bars_u = smem_u32(bars);
  const unsigned q_full = bars_u, kv_full0 = bars_u + 8, kv_empty0 = kv_full0 + 8 * RING, s_full0 = kv_empty0 + 8 * RING,
                 p_full = s_full0 + 16, o_done = p_full + 8;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = (int)gridDim.y - 1 - (int)blockIdx.y, head = blockIdx.x, s = blockIdx.z;
  const int q_len = seq_q_len[s];
  if (tile * BM >= q_len) return;
  if (q_u & 1023u) {
    if (threadIdx.x == 0 && status) atomicExch(status, 40);
    return;
  }
  const int q_start = seq_q_start[s], ctx = seq_ctx_len[s];
  const int seq_row = table_row0 + s;
  const int p0 = ctx - q_len;
  const int kvh = head / (n_heads / pv.n_kv_heads);
  const int rows = min(BM, q_len - tile * BM);
  const int pos_first = p0 + tile * BM, pos_last = pos_first + rows - 1;
  const int lo_first = (window > 0 && pos_first - window + 1 > 0) ? pos_first - window + 1 : 0;
  const int sub0 = lo_first / SUB, n_sub = pos_last / SUB - sub0 + 1;        // sub-tiles of 64 keys

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int st = 0; st < RING; st++) {
      mbar_init(kv_full0 + 8 * st, 1);
      mbar_init(kv_empty0 + 8 * st, 1);
    }
    mbar_init(s_full0, 1);
    mbar_init(s_full0 + 8, 1);
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = *tmem_slot;
  const unsigned tmem_s = tmem_base, tmem_o = tmem_base + 2 * SUB;      // S0, S1: 64 columns each; then O

  if (warp == 4) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      mbar_expect_tx(q_full, Q_BYTES);
      tma_load_2d(q_u, &map_q, head * HD, q_start + tile * BM, q_full);
    }
    for (int j = 0; j < n_sub; j++) {
      const unsigned st = j % RING, round = j / RING;
      // lanes 0..3: the key boxes of the sub-tile's four granules; lanes 4..7: the value boxes
      const int key16 = (sub0 + j) * SUB + (lane & 3) * 16;
      const bool valid = lane < 8 && key16 <= pos_last && key16 + 16 > lo_first;
      int box_row = 0;
      if (valid) {
        const int blk = key16 / pv.page_size;
        const int page = pv.block_table[(long long)seq_row * pv.bt_stride + blk];
        box_row = (page * pv.n_kv_heads + kvh) * pv.page_size + (key16 - blk * pv.page_size);
      }
      const unsigned n_valid = __popc(__ballot_sync(0xffffffffu, valid));
      if (lane == 0) {
        if (round > 0) mbar_wait(kv_empty0 + 8 * st, (round - 1) & 1, status, 41);
        mbar_expect_tx(kv_full0 + 8 * st, n_valid * BOX_BYTES);
      }
      __syncwarp();
      if (valid)
        tma_load_2d(kv_u + st * STAGE_BYTES + (lane >> 2) * K_BYTES + (lane & 3) * BOX_BYTES, lane < 4 ? &map_k : &map_v,
                    0, box_row, kv_full0 + 8 * st);
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------ issuer
    if (lane == 0) {
      const unsigned idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(SUB >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
      const unsigned idesc_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(HD >> 3) << 17) |
                                ((unsigned)(BM >> 4) << 24);
      auto scores = [&](int j) {                   // S[j & 1] = Q K_j^T
        const unsigned st = j % RING;
        mbar_wait(kv_full0 + 8 * st, (j / RING) & 1, status, 43);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned k_addr = kv_u + st * STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < HD / 16; k++)
          umma(tmem_s + (unsigned)((j & 1) * SUB), smem_desc(q_u + k * 32), smem_desc(k_addr + k * 32), idesc_qk,
               k > 0 ? 1u : 0u);
        umma_commit(s_full0 + 8 * (j & 1));
      };
      mbar_wait(q_full, 0, status, 42);
      scores(0);
      if (n_sub > 1) scores(1);
      for (int j = 0; j < n_sub; j++) {
        const unsigned st = j % RING;
        mbar_wait(p_full, j & 1, status, 44);          // P_j is in shared memory, S[j & 1] has been read
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned v_addr = kv_u + st * STAGE_BYTES + K_BYTES;
#pragma unroll
        for (int k = 0; k < SUB / 16; k++)
          umma(tmem_o, smem_desc(p_u + k * 32), smem_desc(v_addr + k * 16 * 128), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(kv_empty0 + 8 * st);               // both products of this stage are behind this
        umma_commit(o_done);
        if (j + 2 < n_sub) scores(j + 2);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax: a query row per thread
    const int r = warp * 32 + lane;
    const unsigned lane_field = (unsigned)(warp * 32) << 16;
    const int my_pos = pos_first + r;
    const int my_lo = (window > 0 && my_pos - window + 1 > 0) ? my_pos - window + 1 : 0;
    const int w_pos_first = pos_first + warp * 32;
    const int w_lo_last = (window > 0 && w_pos_first + 31 - window + 1 > 0) ? w_pos_first + 31 - window + 1 : 0;
    const unsigned p_row = p_u + (r >> 3) * 1024 + (r & 7) * 128;
    float m_row = -INFINITY, l_row = 0.f;
    for (int j = 0; j < n_sub; j++) {
      const int key0 = (sub0 + j) * SUB;
      const unsigned st = j % RING;
      const unsigned s_addr = tmem_s + lane_field + (unsigned)((j & 1) * SUB);
      mbar_wait(s_full0 + 8 * (j & 1), (j >> 1) & 1, status, 45);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const bool edge = key0 + SUB - 1 > w_pos_first || key0 < w_lo_last;
      unsigned sc[2][32];
      float mx = edge ? row_scores_max<true>(s_addr, sc, key0, my_pos, my_lo)
                      : row_scores_max<false>(s_addr, sc, key0, my_pos, my_lo);
      mx *= scale_log2;
      const float m_cand = fmaxf(m_row, mx);
      // also from -inf; rows past the portion (another's queries, keys that were not fetched) have no say in it
      const bool moved = __any_sync(0xffffffffu, r < rows && m_cand - m_row > MAX_SLACK_LOG2);
      const float m_new = moved ? m_cand : m_row;
      const float m_off = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = !moved ? 1.f : ((m_row == -INFINITY) ? 0.f : ex2(m_row - m_off));
      if (j > 0) {                                   // O += P V of the sub-tile before: P is free, O is whole
        mbar_wait(o_done, (j - 1) & 1, status, 46);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (moved) {
#pragma unroll 1
          for (int c = 0; c < HD / 32; c++) {
            float v[32];
            tmem_ld32(tmem_o + lane_field + (unsigned)(c * 32), v);
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] *= alpha;
            tmem_st32(tmem_o + lane_field + (unsigned)(c * 32), v);
          }
        }
      }
      if (key0 + SUB - 1 > pos_last || key0 < lo_first) {      // value rows of keys no query may see (thread = key)
        const int key = key0 + r;
        if (r < SUB && (key > pos_last || key < lo_first)) {
          const unsigned row_u = kv_u + st * STAGE_BYTES + K_BYTES + r * 128;
#pragma unroll
          for (int c = 0; c < 8; c++) sts128(row_u + c * 16, 0u, 0u, 0u, 0u);
        }
      }
      const float sum = row_probabilities(sc, p_row, r, scale_log2, m_off);
      l_row = l_row * alpha + sum;
      m_row = m_new;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    mbar_wait(o_done, (n_sub - 1) & 1, status, 47);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const float inv = 1.0f / l_row;
    __nv_bfloat16* orow = out + ((long long)(q_start + tile * BM + r) * n_heads + head) * HD;
#pragma unroll 1
    for (int c = 0; c < HD / 32; c++) {
      float v[32];
      tmem_ld32(tmem_o + lane_field + (unsigned)(c * 32), v);
      if (r < rows) {
#pragma unroll
        for (int q4 = 0; q4 < 4; q4++) {
          uint4 pk;
          pk.x = pack_bf16(v[q4 * 8 + 0] * inv, v[q4 * 8 + 1] * inv);
          pk.y = pack_bf16(v[q4 * 8 + 2] * inv, v[q4 * 8 + 3] * inv);
          pk.z = pack_bf16(v[q4 * 8 + 4] * inv, v[q4 * 8 + 5] * inv);
          pk.w = pack_bf16(v[q4 * 8 + 6] * inv, v[q4 * 8 + 7] * inv);
          *reinterpret_cast<uint4*>(orow + c * 32 + q4 * 8) = pk;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS));
  }
}

int launch_tc_ahead(const __nv_bfloat16* q, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool, __nv_bfloat16* out,
                    const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len, int table_row0, int n_seqs,
                    int max_q_len, int n_tokens, int n_heads, PagedView pv, float scale, int window, int* status,
                    cudaStream_t stream) {
  CUtensorMap mq, mk, mv;
  int rc = tma_host::bf16_map(q, n_tokens, (long long)n_heads * ahead::HD, BM, 64, &mq);
  if (rc) return rc;
  rc = tma_host::bf16_map(k_pool, pv.pool_rows, ahead::HD, 16, 64, &mk);
  if (rc) return rc;
  rc = tma_host::bf16_map(v_pool, pv.pool_rows, ahead::HD, 16, 64, &mv);
  if (rc) return rc;
  static DeviceOnce once;
  const int dev_ = mf_current_device();
  if (dev_ < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev_]) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_ahead_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)ahead::SMEM);
    if (e != cudaSuccess) return (int)e;
    once.done[dev_] = true;
  }
  dim3 grid(n_heads, (max_q_len + BM - 1) / BM, n_seqs);
  mf_count(MF_K_ATTN_PREFILL_TC);
  attn_prefill_tc_ahead_kernel<<<grid, 192, ahead::SMEM, stream>>>(mq, mk, mv, out, seq_q_start, seq_q_len, seq_ctx_len,
                                                                   table_row0, pv, n_heads, scale * LOG2E, window, status);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Head size 128 (with or without options) and attention whose values are the first channels of its keys (a latent that all query
// heads share: keys of up to 256 channels, values of up to 192): TWO CHAINS a block.  A block's 128 queries walk their keys by
// pairs of tiles of 64; the first tile of a pair belongs to one group of four softmax warps, the second to another, and a group
// has a result, a running maximum and a sum of its own.  The two results are joined at the end as two splits of the keys are.
//   warps 0-3   the softmax of the first tiles, warps 4-7 of the second ones (a query row per thread)
//   warp 8      producer: a stage is a pair of tiles of keys and of values (those by warp 10); where the values lie in the keys,
//               the keys alone, read along their channels by S = Q K^T and as the N-major operand by O += P V
//   warp 9      issuer of S of both tiles as one product (N 128), for pair j + 1 as soon as the warps have S of pair j in registers
//   warp 11     issuer of O += P V, a product for each chain over all the values' columns
// Why (a block's clock, stamped at every hand-over): with one chain and one producer warp a tile took 1.7 us in a block with the SM to
// itself, whatever the softmax did.  (1) A tensor copy takes the issuing warp 67 cycles, 1,070 for the sixteen granules of a tile of
// 2 x 2 spans: a tile whose four pages follow one another is one copy a span.  (2) Scores waited for keys behind values that waited for
// a product: keys and values have producers and stages of their own.  (3) One issuing thread held a finished P back while it waited
// for the next keys: S and O += P V have an issuer each.  (4) A product of N 64 takes 60 to 73 cycles a step of K 16, as long as
// its operands take to come from shared memory, one of N 128 or 192 hardly more, so products are as wide as they can be and P
// stays in tensor memory where there is room.  (5) The block with the most keys decides: its keys go through two chains.
// What is left is the softmax's own chain of instructions, 2,700 cycles a pair (1,024 of them the exponentials' unit).
// Measured: 16 heads of 128 with a window, three prompts of 2,237 tokens, 54 -> 37 us (the layer 112.7 -> 98.5); one head's 2,048
// tokens 41 -> 29 (rescaled at every move of a maximum), 400 tokens of two 32-head sequences behind 500 keys 22 -> 13.6; 16 heads over a
// latent of 192 + 32 channels, 2,048 tokens, 64 -> 51 (the layer 136 -> 122): there a pair of tiles is 56 KB of keys, read twice
// and from the one pair of stages that fits, so the copies are part of the chain.
// A latent head that is no whole number of 64-wide spans leaves the last span's rest to the next head's channels or to zeros; the
// products' steps of 16 channels end before it.
namespace pair {
constexpr int SUB = 64, P_BYTES = BM * SUB * 2, K_SPAN_BYTES = 2 * SUB * 128, Q_SPAN_BYTES = BM * 128;
constexpr int stage_spans(int spans, int vspans, bool own_v) { return spans + (own_v ? vspans : 0); }
constexpr int ring(int stage_spans) { return stage_spans == 4 ? 2 : 3; }
constexpr int THREADS = 384;
// P as the A operand in tensor memory where two results leave room for it: neither written to nor read from shared memory
constexpr bool p_in_tmem(int vspans) { return 2 * SUB + 2 * vspans * 64 + SUB <= 512; }
// N-major operand of several 64-wide spans: a span's lines are K_SPAN_BYTES from the next span's
__device__ __forceinline__ unsigned long long values_desc(unsigned addr) {
  return (smem_desc(addr) & ~((unsigned long long)0x3FFF << 16)) | (unsigned long long)(K_SPAN_BYTES >> 4) << 16;
}
constexpr size_t smem(int spans, int vspans, bool own_v) {
  const int st = stage_spans(spans, vspans, own_v);
  return (size_t)spans * Q_SPAN_BYTES + (size_t)ring(st) * st * K_SPAN_BYTES + 2 * P_BYTES + 24 * 8 + 16;
}
__device__ __forceinline__ void group_sync() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }
// columns of tensor memory times a number per row; the stores are waited for at the end
__device__ __forceinline__ void scale_columns(unsigned taddr, int cols, float by) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 32) {
    float v[32];
    tmem_ld32(taddr + (unsigned)c, v);
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] *= by;
    tmem_st32_issue(taddr + (unsigned)c, v);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}
}  // namespace pair

template <int SPANS, int VSPANS, bool OWN_V, bool EX>
__global__ void __launch_bounds__(pair::THREADS, 1)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_k4,
                         const __grid_constant__ CUtensorMap map_v4, __nv_bfloat16* __restrict__ out,
                         const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len,
                         const int* __restrict__ seq_ctx_len, int table_row0, PagedView pv, int n_heads, int vd,
                         float scale_log2, int window, int* __restrict__ status, const TcOptions opt) {
  using namespace pair;
  constexpr int ST = stage_spans(SPANS, VSPANS, OWN_V), RING = ring(ST), STAGE_BYTES = ST * K_SPAN_BYTES;
  constexpr int Q_BYTES = SPANS * Q_SPAN_BYTES, V_OFF = OWN_V ? SPANS * K_SPAN_BYTES : 0, VCOLS = VSPANS * 64;
  constexpr bool P_IN_TMEM = p_in_tmem(VSPANS);
  constexpr int USED = 2 * SUB + 2 * VCOLS + (P_IN_TMEM ? SUB : 0), COLS = USED <= 256 ? 256 : 512;
  static_assert(USED <= 512, "two chains share the tensor memory");
  static_assert(VCOLS / 2 * BM * 2 * 4 <= Q_BYTES + RING * STAGE_BYTES, "halves of both results are traded through shared memory");
  extern __shared__ __align__(1024) unsigned char smem[];
  const unsigned q_u = smem_u32(smem), kv_u = q_u + Q_BYTES, p_u = kv_u + RING * STAGE_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + Q_BYTES + RING * STAGE_BYTES + 2 * P_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 24);
  __shared__ float2 ml_s[2][BM];
  const unsigned bars_u = smem_u32(bars);
  // of keys and of values apart, where they are: keys are free again once S is made
  const unsigned q_full = bars_u, k_full0 = bars_u + 8, k_empty0 = k_full0 + 8 * RING, v_full0 = k_empty0 + 8 * RING,
                 v_empty0 = v_full0 + 8 * RING, s_full = v_empty0 + 8 * RING, s_free = s_full + 8, p_full0 = s_free + 8,
                 o_done0 = p_full0 + 16;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the heaviest tiles (the last queries of a portion see the most keys) of all sequences and heads are launched first
  const int tile = (int)gridDim.z - 1 - (int)blockIdx.z, head = blockIdx.x, s = blockIdx.y;
  const int q_len = seq_q_len[s];
  if (tile * BM >= q_len || (EX && q_len < opt.min_len)) return;
  if (q_u & 1023u) {                                       // never seen; refused rather than computed wrongly
    if (threadIdx.x == 0 && status) atomicExch(status, 40);
    return;
  }
  const int hd = pv.head_dim;
  const int q_start = seq_q_start[s], ctx = seq_ctx_len[s];
  const int seq_row = table_row0 + s;
  const int p0 = ctx - q_len;                              // position of the portion's first token
  const int kvh = head / (n_heads / pv.n_kv_heads);
  const int rows = min(BM, q_len - tile * BM);             // valid queries in this tile
  const int pos_first = p0 + tile * BM, pos_last = pos_first + rows - 1;
  const int lo_first = (window > 0 && pos_first - window + 1 > 0) ? pos_first - window + 1 : 0;
  const int kt0 = lo_first / SUB, kt1 = pos_last / SUB;    // key tiles [kt0, kt1]
  const int keep = EX && window > 0 ? opt.keep_first : 0;
  const int n_kept = EX ? min((keep + SUB - 1) / SUB, kt0) : 0;                // tiles of kept keys before them
  const int n_kt = kt1 - kt0 + 1 + n_kept, n_pairs = (n_kt + 1) / 2;
  auto tile_of = [&](int i) { return EX && i < n_kept ? i : kt0 + i - n_kept; };

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int st = 0; st < RING; st++) {
      mbar_init(k_full0 + 8 * st, 1);
      mbar_init(k_empty0 + 8 * st, 1);
      mbar_init(v_full0 + 8 * st, 1);
      mbar_init(v_empty0 + 8 * st, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, 8);                           // one arrive per softmax warp
    for (int c = 0; c < 2; c++) {
      mbar_init(p_full0 + 8 * c, 4);                // one arrive per softmax warp of the chain
      mbar_init(o_done0 + 8 * c, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = *tmem_slot;                   // S of a pair: 64 columns a chain; then the chains' O

  if (warp == 8 || (OWN_V && warp == 10)) {
    // ------------------------------------------------------------ producers: of the keys, of the values
    const bool values = warp == 10;
    if (!values) {
      if (lane == 0) mbar_expect_tx(q_full, Q_BYTES);      // rows past the end of q arrive as zeros
      __syncwarp();
      if (lane < SPANS) tma_load_2d(q_u + lane * Q_SPAN_BYTES, &map_q, head * hd + lane * 64, q_start + tile * BM, q_full);
    }
    const int spans = values ? VSPANS : SPANS;
    const unsigned full0 = values ? v_full0 : k_full0, empty0 = values ? v_empty0 : k_empty0;
    const CUtensorMap* map1 = values ? &map_v : &map_k;
    const CUtensorMap* map4 = values ? &map_v4 : &map_k4;
    // A lane per granule of 16 keys and span; a granule with no visible key is not fetched (-1).  Its page is looked up a pair
    // ahead, so that no copy waits for the table.  The unit takes about 67 cycles to accept a copy, whatever its size: a tile
    // whose four granules are pages that follow one another (pages of 16 tokens; a fresh cache gives a sequence such pages)
    // comes as one copy a span.
    const int gran = lane & 7, span = lane >> 3;
    auto page_of = [&](int j) {
      const int i = 2 * j + (gran >> 2), key16 = tile_of(i) * SUB + (gran & 3) * 16;
      if (j >= n_pairs || span >= spans || i >= n_kt || key16 > pos_last || !(key16 + 16 > lo_first || (EX && key16 < keep))) return -1;
      return pv.block_table[(long long)seq_row * pv.bt_stride + (pv.page_size == 16 ? key16 >> 4 : key16 / pv.page_size)];
    };
    int page = page_of(0);
    for (int j = 0; j < n_pairs; j++) {
      const unsigned st = j % RING;
      const int next = page_of(j + 1);
      const bool valid = page >= 0;
      const int first = __shfl_sync(0xffffffffu, page, lane & ~3);
      const unsigned follows = __ballot_sync(0xffffffffu, valid && first >= 0 && page == first + (gran & 3));
      const bool run = pv.page_size == 16 && (follows >> (lane & ~3) & 15) == 15;
      const unsigned n_valid = __popc(__ballot_sync(0xffffffffu, valid));
      if (lane == 0) {
        if (j >= RING) mbar_wait(empty0 + 8 * st, (j / RING - 1) & 1, status, 41);
        mbar_expect_tx(full0 + 8 * st, n_valid * BOX_BYTES);
      }
      __syncwarp();
      const unsigned dst = kv_u + st * STAGE_BYTES + (values ? V_OFF : 0) + span * K_SPAN_BYTES + gran * BOX_BYTES;
      if (run) {
        if ((gran & 3) == 0) tma_load_3d(dst, map4, span * 64, kvh * 16, page, full0 + 8 * st);
      } else if (valid) {
        const int key16 = tile_of(2 * j + (gran >> 2)) * SUB + (gran & 3) * 16;
        tma_load_2d(dst, map1, span * 64, (page * pv.n_kv_heads + kvh) * pv.page_size + key16 % pv.page_size, full0 + 8 * st);
      }
      page = next;
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------ issuer of S = Q K^T of both tiles of a pair
    if (lane == 0) {
      // instruction descriptor: D float32, A and B bfloat16; N >> 3 at bit 17, M >> 4 at bit 24
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(2 * SUB >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
      const int steps = OWN_V ? SPANS * 4 : hd / 16;
      const unsigned long long q_desc = smem_desc(q_u);
      mbar_wait(q_full, 0, status, 42);
      for (int j = 0; j < n_pairs; j++) {
        const unsigned st = j % RING;
        const unsigned long long k_desc = smem_desc(kv_u + st * STAGE_BYTES);
        mbar_wait(k_full0 + 8 * st, (j / RING) & 1, status, 43);
        if (j > 0) mbar_wait(s_free, (j - 1) & 1, status, 48);         // S of the pair before is in registers
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
        for (int k = 0; k < SPANS * 4; k++)
          if (OWN_V || k < steps)
            umma(tmem_base, q_desc + (((k >> 2) * Q_SPAN_BYTES + (k & 3) * 32) >> 4),
                 k_desc + (((k >> 2) * K_SPAN_BYTES + (k & 3) * 32) >> 4), idesc, k > 0 ? 1u : 0u);
        umma_commit(s_full);
        if (OWN_V) umma_commit(k_empty0 + 8 * st);
      }
    }
  } else if (warp == 11) {
    // ------------------------------------------------------------ issuer of O += P V, chain by chain
    if (lane == 0) {
      // bit 16: B is N-major (the values)
      const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(VCOLS >> 3) << 17) |
                             ((unsigned)(BM >> 4) << 24);
      for (int j = 0; j < n_pairs; j++) {
        const unsigned st = j % RING;
        if (OWN_V) mbar_wait(v_full0 + 8 * st, (j / RING) & 1, status, 49);
#pragma unroll
        for (int c = 0; c < 2; c++) {
          if (2 * j + c >= n_kt) break;
          const unsigned long long v_desc = values_desc(kv_u + st * STAGE_BYTES + V_OFF + c * SUB * 128);
          const unsigned long long p_desc = smem_desc(p_u + c * P_BYTES);
          const unsigned tmem_o = tmem_base + (unsigned)(2 * SUB + c * VCOLS), tmem_p = tmem_base + (unsigned)(2 * SUB + 2 * VCOLS + c * 32);
          mbar_wait(p_full0 + 8 * c, j & 1, status, 44);               // P is there
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
          for (int k = 0; k < SUB / 16; k++)
            if (P_IN_TMEM)
              umma_ta(tmem_o, tmem_p + (unsigned)(k * 8), v_desc + (k * 16 * 128 >> 4), idesc, (j > 0 || k > 0) ? 1u : 0u);
            else
              umma(tmem_o, p_desc + (k * 32 >> 4), v_desc + (k * 16 * 128 >> 4), idesc, (j > 0 || k > 0) ? 1u : 0u);
          umma_commit(o_done0 + 8 * c);
        }
        // all products of this stage are behind this: P comes of S
        umma_commit((OWN_V ? v_empty0 : k_empty0) + 8 * st);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ softmax: a query row per thread
    const int chain = warp >> 2, r = (warp & 3) * 32 + lane;
    const unsigned lane_field = (unsigned)((warp & 3) * 32) << 16;
    const unsigned tmem_s = tmem_base + lane_field + (unsigned)(chain * SUB);
    const unsigned tmem_o = tmem_base + lane_field + (unsigned)(2 * SUB + chain * VCOLS);
    const unsigned tmem_p = tmem_base + lane_field + (unsigned)(2 * SUB + 2 * VCOLS + chain * 32);
    const unsigned p_full = p_full0 + 8 * chain, o_done = o_done0 + 8 * chain;
    const int my_pos = pos_first + r;
    const int my_lo = (window > 0 && my_pos - window + 1 > 0) ? my_pos - window + 1 : 0;
    const int w_pos_first = pos_first + (warp & 3) * 32;    // this warp's first query
    const int w_lo_last = (window > 0 && w_pos_first + 31 - window + 1 > 0) ? w_pos_first + 31 - window + 1 : 0;
    const unsigned p_row = p_u + chain * P_BYTES + (r >> 3) * 1024 + (r & 7) * 128;
    float m_row = -INFINITY, l_row = 0.f;
    if (EX && opt.sink && chain == 0) {     // a key of this score whose value is zero
      m_row = opt.sink[head] * LOG2E;
      l_row = 1.f;
    }
    int n = 0;                              // tiles of this chain behind: the pair
    for (int i = chain; i < n_kt; i += 2, n++) {
      const int key0 = tile_of(i) * SUB;
      const unsigned st = n % RING;
      mbar_wait(s_full, n & 1, status, 45);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      // mask only where the tile touches this warp's diagonal or an end of its windows
      const bool edge = key0 + SUB - 1 > w_pos_first || key0 < w_lo_last;
      // ---- first pass over the row of S: its maximum
      unsigned sc[2][32];
      float mx = edge ? row_scores_max<true>(tmem_s, sc, key0, my_pos, my_lo, keep)
                      : row_scores_max<false>(tmem_s, sc, key0, my_pos, my_lo);
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);
      mx *= scale_log2;                                      // scale > 0: the max commutes with it
      const float m_cand = fmaxf(m_row, mx);
      // also from -inf; rows past the portion (another's queries, keys that were not fetched) have no say in it
      const bool moved = __any_sync(0xffffffffu, r < rows && m_cand - m_row > (EX ? EXACT_MAX_LOG2 : MAX_SLACK_LOG2));
      const float m_new = moved ? m_cand : m_row;
      const float m_off = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = !moved ? 1.f : ((m_row == -INFINITY) ? 0.f : ex2(m_row - m_off));
      // ---- the product before this one has read P and left O: rescale O if a maximum moved
      if (n > 0) {
        mbar_wait(o_done, (n - 1) & 1, status, 46);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (moved) scale_columns(tmem_o, VCOLS, alpha);
      }
      // ---- value rows of keys that no query of the tile may see: clear them (thread = key) once they are there (where they lie in
      // the keys: S of the tile is made, so they are)
      if (key0 + SUB - 1 > pos_last || key0 < lo_first) {
        if (OWN_V) mbar_wait(v_full0 + 8 * st, (n / RING) & 1, status, 50);
        const int key = key0 + r;
        if (r < SUB && (key > pos_last || (key < lo_first && key >= keep))) {
#pragma unroll
          for (int sp = 0; sp < VSPANS; sp++) {
            const unsigned row_u = kv_u + st * STAGE_BYTES + V_OFF + sp * K_SPAN_BYTES + (chain * SUB + r) * 128;
#pragma unroll
            for (int c = 0; c < 8; c++) sts128(row_u + c * 16, 0u, 0u, 0u, 0u);
          }
        }
      }
      // ---- second pass: probabilities, their sum, and the row of P in the operand layout
      const float sum = P_IN_TMEM ? row_probabilities_tmem(sc, tmem_p, scale_log2, m_off)
                                  : row_probabilities(sc, p_row, r, scale_log2, m_off);
      l_row = l_row * alpha + sum;
      m_row = m_new;
      // P and the cleared rows, before the product reads them from shared memory
      if (!P_IN_TMEM || key0 + SUB - 1 > pos_last || key0 < lo_first) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    // ---- the two results joined: a group keeps half of the columns of its own and is given the other group's
    if (n > 0) {
      mbar_wait(o_done, (n - 1) & 1, status, 47);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    constexpr int HALF = VCOLS / 2;
    const bool mine_counts = n > 0 && m_row != -INFINITY;
    ml_s[chain][r] = make_float2(n > 0 || m_row != -INFINITY ? m_row : -INFINITY, l_row);
    group_sync();            // all products are done: what the queries and stages stood in is free
    // [group given to][columns by four][row]: 16-byte pieces of neighbouring rows side by side
    float4* give = reinterpret_cast<float4*>(smem) + (chain ^ 1) * (HALF / 4) * BM + r;
    const float4* take = reinterpret_cast<const float4*>(smem) + chain * (HALF / 4) * BM + r;
    if (n > 0) {
#pragma unroll 1
      for (int c = 0; c < HALF; c += 32) {
        float v[32];
        tmem_ld32(tmem_o + (unsigned)((chain ^ 1) * HALF + c), v);
#pragma unroll
        for (int j = 0; j < 32; j += 4) give[(c + j) / 4 * BM] = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
    }
    group_sync();
    const float2 other = ml_s[chain ^ 1][r];
    const bool other_counts = n_kt > (chain ^ 1) && other.x != -INFINITY;
    const float m = fmaxf(m_row, other.x);
    const float w_mine = m_row == -INFINITY ? 0.f : ex2(m_row - m), w_other = other.x == -INFINITY ? 0.f : ex2(other.x - m);
    const float inv = 1.0f / (l_row * w_mine + other.y * w_other);
    const float f_mine = w_mine * inv, f_other = w_other * inv;
    __nv_bfloat16* orow = out + ((long long)(q_start + tile * BM + r) * n_heads + head) * vd;
#pragma unroll 1
    for (int c = 0; c < HALF; c += 32) {
      const int col = chain * HALF + c;
      float v[32];
      if (n > 0) {
        tmem_ld32(tmem_o + (unsigned)col, v);
      } else {
#pragma unroll
        for (int j = 0; j < 32; j++) v[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 x = other_counts ? take[(c + j) / 4 * BM] : make_float4(0.f, 0.f, 0.f, 0.f);
        v[j] = (mine_counts ? v[j] * f_mine : 0.f) + x.x * f_other;
        v[j + 1] = (mine_counts ? v[j + 1] * f_mine : 0.f) + x.y * f_other;
        v[j + 2] = (mine_counts ? v[j + 2] * f_mine : 0.f) + x.z * f_other;
        v[j + 3] = (mine_counts ? v[j + 3] * f_mine : 0.f) + x.w * f_other;
      }
      if (r < rows) {
#pragma unroll
        for (int q4 = 0; q4 < 4; q4++) {
          if (!OWN_V && col + q4 * 8 >= vd) continue;
          if (EX && OWN_V && opt.gate)
            apply_gate(v + q4 * 8, opt.gate + (long long)(q_start + tile * BM + r) * opt.gate_ld + head * vd + col + q4 * 8);
          uint4 pk;
          pk.x = pack_bf16(v[q4 * 8 + 0], v[q4 * 8 + 1]);
          pk.y = pack_bf16(v[q4 * 8 + 2], v[q4 * 8 + 3]);
          pk.z = pack_bf16(v[q4 * 8 + 4], v[q4 * 8 + 5]);
          pk.w = pack_bf16(v[q4 * 8 + 6], v[q4 * 8 + 7]);
          *reinterpret_cast<uint4*>(orow + col + q4 * 8) = pk;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 9) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(COLS));
  }
}

template <int SPANS, int VSPANS, bool OWN_V, bool EX>
int launch_pair(const __nv_bfloat16* q, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool, __nv_bfloat16* out,
                const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len, int table_row0, int n_seqs,
                int max_q_len, int n_tokens, int n_heads, PagedView pv, int vd, float scale, int window, int* status,
                const TcOptions& opt, cudaStream_t stream) {
  CUtensorMap mq, mk, mv, mk4, mv4;
  int rc = tma_host::bf16_map(q, n_tokens, (long long)n_heads * pv.head_dim, BM, 64, &mq);
  if (rc) return rc;
  rc = tma_host::bf16_map(k_pool, pv.pool_rows, pv.head_dim, 16, 64, &mk);
  if (rc) return rc;
  if (OWN_V) {
    rc = tma_host::bf16_map(v_pool, pv.pool_rows, vd, 16, 64, &mv);
    if (rc) return rc;
  } else {
    mv = mk;
  }
  // four pages of 16 tokens at once: [pages][rows of a page][channels]
  mk4 = mk, mv4 = mv;
  if (pv.page_size == 16) {
    const long long pages = pv.pool_rows / (pv.n_kv_heads * 16);
    rc = tma_host::bf16_map_pages(k_pool, pages, pv.n_kv_heads * 16, pv.head_dim, 4, &mk4);
    if (rc) return rc;
    rc = OWN_V ? tma_host::bf16_map_pages(v_pool, pages, pv.n_kv_heads * 16, vd, 4, &mv4) : 0;
    if (rc) return rc;
  }
  constexpr size_t smem = pair::smem(SPANS, VSPANS, OWN_V);
  static DeviceOnce once;
  const int dev_ = mf_current_device();
  if (dev_ < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev_]) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_pair_kernel<SPANS, VSPANS, OWN_V, EX>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev_] = true;
  }
  const dim3 grid(n_heads, n_seqs, (max_q_len + BM - 1) / BM);
  mf_count(MF_K_ATTN_PREFILL_TC);
  if (!OWN_V) mf_count(MF_K_ATTN_PREFILL_LATENT);
  attn_prefill_pair_kernel<SPANS, VSPANS, OWN_V, EX><<<grid, pair::THREADS, smem, stream>>>(
      mq, mk, mv, mk4, mv4, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, pv, n_heads, vd, scale * LOG2E, window, status, opt);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Latents whose values are wider than 192 channels, whose two results would not fit in tensor memory: the kernel for head size 64
// with a wider head, products ahead of the softmax, two S buffers, O behind them; a stage is ONE tile of 64 keys, read once along its
// channels by S = Q K^T and once as the N-major operand by O += P V.  One block per SM (the queries' tile alone is 64 KB).
namespace latent {
constexpr int SUB = 64, P_BYTES = BM * SUB * 2, K_SPAN_BYTES = SUB * 128, Q_SPAN_BYTES = BM * 128;
constexpr int ring(int spans) { return spans == 4 ? 4 : 5; }
constexpr size_t smem(int spans) {
  return (size_t)spans * Q_SPAN_BYTES + (size_t)ring(spans) * spans * K_SPAN_BYTES + P_BYTES + 24 * 8 + 16;
}
}  // namespace latent

template <int SPANS, int VSPANS>
__global__ void __launch_bounds__(192, 1)
attn_prefill_latent_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           __nv_bfloat16* __restrict__ out, const int* __restrict__ seq_q_start,
                           const int* __restrict__ seq_q_len, const int* __restrict__ seq_ctx_len, int table_row0, PagedView pv,
                           int n_heads, int vd, float scale_log2, int window, int min_len, int* __restrict__ status) {
  using namespace latent;
  constexpr int RING = ring(SPANS), STAGE_BYTES = SPANS * K_SPAN_BYTES, Q_BYTES = SPANS * Q_SPAN_BYTES;
  constexpr int COLS = 2 * SUB + VSPANS * 64 <= 256 ? 256 : 512;
  extern __shared__ __align__(1024) unsigned char smem[];
  const unsigned q_u = smem_u32(smem), kv_u = q_u + Q_BYTES, p_u = kv_u + RING * STAGE_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + Q_BYTES + RING * STAGE_BYTES + P_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 24);
  const unsigned bars_u = smem_u32(bars);
  const unsigned q_full = bars_u, kv_full0 = bars_u + 8, kv_empty0 = kv_full0 + 8 * RING, s_full0 = kv_empty0 + 8 * RING,
                 p_full = s_full0 + 16, o_done = p_full + 8;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = (int)gridDim.y - 1 - (int)blockIdx.y, head = blockIdx.x, s = blockIdx.z;
  const int q_len = seq_q_len[s];
  if (tile * BM >= q_len || q_len < min_len) return;
  if (q_u & 1023u) {
    if (threadIdx.x == 0 && status) atomicExch(status, 40);
    return;
  }
  const int hd = pv.head_dim;
  const int q_start = seq_q_start[s], ctx = seq_ctx_len[s];
  const int seq_row = table_row0 + s;
  const int p0 = ctx - q_len;
  const int kvh = head / (n_heads / pv.n_kv_heads);
  const int rows = min(BM, q_len - tile * BM);
  const int pos_first = p0 + tile * BM, pos_last = pos_first + rows - 1;
  const int lo_first = (window > 0 && pos_first - window + 1 > 0) ? pos_first - window + 1 : 0;
  const int sub0 = lo_first / SUB, n_sub = pos_last / SUB - sub0 + 1;        // tiles of 64 keys

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int st = 0; st < RING; st++) {
      mbar_init(kv_full0 + 8 * st, 1);
      mbar_init(kv_empty0 + 8 * st, 1);
    }
    mbar_init(s_full0, 1);
    mbar_init(s_full0 + 8, 1);
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = *tmem_slot;
  const unsigned tmem_s = tmem_base, tmem_o = tmem_base + 2 * SUB;      // S0, S1: 64 columns each; then O

  if (warp == 4) {
    // ------------------------------------------------------------ producer
    if (lane == 0) mbar_expect_tx(q_full, Q_BYTES);
    __syncwarp();
    if (lane < SPANS) tma_load_2d(q_u + lane * Q_SPAN_BYTES, &map_q, head * hd + lane * 64, q_start + tile * BM, q_full);
    for (int j = 0; j < n_sub; j++) {
      const unsigned st = j % RING, round = j / RING;
      // a lane per granule of 16 keys and span
      const int gran = lane & 3, span = lane >> 2;
      const int key16 = (sub0 + j) * SUB + gran * 16;
      const bool valid = span < SPANS && key16 <= pos_last && key16 + 16 > lo_first;
      int box_row = 0;
      if (valid) {
        const int blk = key16 / pv.page_size;
        const int page = pv.block_table[(long long)seq_row * pv.bt_stride + blk];
        box_row = (page * pv.n_kv_heads + kvh) * pv.page_size + (key16 - blk * pv.page_size);
      }
      const unsigned n_valid = __popc(__ballot_sync(0xffffffffu, valid));
      if (lane == 0) {
        if (round > 0) mbar_wait(kv_empty0 + 8 * st, (round - 1) & 1, status, 41);
        mbar_expect_tx(kv_full0 + 8 * st, n_valid * BOX_BYTES);
      }
      __syncwarp();
      if (valid)
        tma_load_2d(kv_u + st * STAGE_BYTES + span * K_SPAN_BYTES + gran * BOX_BYTES, &map_k, span * 64, box_row,
                    kv_full0 + 8 * st);
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------ issuer
    if (lane == 0) {
      const unsigned idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(SUB >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
      const unsigned idesc_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(64 >> 3) << 17) |
                                ((unsigned)(BM >> 4) << 24);
      const int steps = hd / 16;
      auto scores = [&](int j) {                   // S[j & 1] = Q K_j^T
        const unsigned st = j % RING;
        mbar_wait(kv_full0 + 8 * st, (j / RING) & 1, status, 43);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned k_addr = kv_u + st * STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < SPANS * 4; k++)
          if (k < steps)
            umma(tmem_s + (unsigned)((j & 1) * SUB), smem_desc(q_u + (k >> 2) * Q_SPAN_BYTES + (k & 3) * 32),
                 smem_desc(k_addr + (k >> 2) * K_SPAN_BYTES + (k & 3) * 32), idesc_qk, k > 0 ? 1u : 0u);
        umma_commit(s_full0 + 8 * (j & 1));
      };
      mbar_wait(q_full, 0, status, 42);
      scores(0);
      if (n_sub > 1) scores(1);
      for (int j = 0; j < n_sub; j++) {
        const unsigned st = j % RING;
        mbar_wait(p_full, j & 1, status, 44);          // P_j is in shared memory, S[j & 1] has been read
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned v_addr = kv_u + st * STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < SUB / 16; k++)
#pragma unroll
          for (int sp = 0; sp < VSPANS; sp++)
            umma(tmem_o + (unsigned)(sp * 64), smem_desc(p_u + k * 32), smem_desc(v_addr + sp * K_SPAN_BYTES + k * 16 * 128),
                 idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(kv_empty0 + 8 * st);               // both products of this stage are behind this
        umma_commit(o_done);
        if (j + 2 < n_sub) scores(j + 2);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax: a query row per thread
    const int r = warp * 32 + lane;
    const unsigned lane_field = (unsigned)(warp * 32) << 16;
    const int my_pos = pos_first + r;
    const int my_lo = (window > 0 && my_pos - window + 1 > 0) ? my_pos - window + 1 : 0;
    const int w_pos_first = pos_first + warp * 32;
    const int w_lo_last = (window > 0 && w_pos_first + 31 - window + 1 > 0) ? w_pos_first + 31 - window + 1 : 0;
    const unsigned p_row = p_u + (r >> 3) * 1024 + (r & 7) * 128;
    float m_row = -INFINITY, l_row = 0.f;
    for (int j = 0; j < n_sub; j++) {
      const int key0 = (sub0 + j) * SUB;
      const unsigned st = j % RING;
      const unsigned s_addr = tmem_s + lane_field + (unsigned)((j & 1) * SUB);
      mbar_wait(s_full0 + 8 * (j & 1), (j >> 1) & 1, status, 45);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const bool edge = key0 + SUB - 1 > w_pos_first || key0 < w_lo_last;
      unsigned sc[2][32];
      float mx = edge ? row_scores_max<true>(s_addr, sc, key0, my_pos, my_lo)
                      : row_scores_max<false>(s_addr, sc, key0, my_pos, my_lo);
      mx *= scale_log2;
      const float m_cand = fmaxf(m_row, mx);
      const bool moved = __any_sync(0xffffffffu, m_cand - m_row > EXACT_MAX_LOG2);      // also from -inf
      const float m_new = moved ? m_cand : m_row;
      const float m_off = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = !moved ? 1.f : ((m_row == -INFINITY) ? 0.f : ex2(m_row - m_off));
      if (j > 0) {                                   // O += P V of the tile before: P is free, O is whole
        mbar_wait(o_done, (j - 1) & 1, status, 46);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (moved) {
#pragma unroll 1
          for (int c = 0; c < VSPANS * 2; c++) {
            float v[32];
            tmem_ld32(tmem_o + lane_field + (unsigned)(c * 32), v);
#pragma unroll
            for (int i = 0; i < 32; i++) v[i] *= alpha;
            tmem_st32(tmem_o + lane_field + (unsigned)(c * 32), v);
          }
        }
      }
      // rows of keys no query may see, before they are read as values (S of the tile is made: nothing else reads them)
      if (key0 + SUB - 1 > pos_last || key0 < lo_first) {
        const int key = key0 + r;
        if (r < SUB && (key > pos_last || key < lo_first)) {
#pragma unroll
          for (int sp = 0; sp < VSPANS; sp++) {
            const unsigned row_u = kv_u + st * STAGE_BYTES + sp * K_SPAN_BYTES + r * 128;
#pragma unroll
            for (int c = 0; c < 8; c++) sts128(row_u + c * 16, 0u, 0u, 0u, 0u);
          }
        }
      }
      const float sum = row_probabilities(sc, p_row, r, scale_log2, m_off);
      l_row = l_row * alpha + sum;
      m_row = m_new;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    mbar_wait(o_done, (n_sub - 1) & 1, status, 47);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const float inv = 1.0f / l_row;
    __nv_bfloat16* orow = out + ((long long)(q_start + tile * BM + r) * n_heads + head) * vd;
#pragma unroll 1
    for (int c = 0; c < VSPANS * 2; c++) {
      float v[32];
      tmem_ld32(tmem_o + lane_field + (unsigned)(c * 32), v);
      if (r < rows) {
#pragma unroll
        for (int q4 = 0; q4 < 4; q4++) {
          if (c * 32 + q4 * 8 < vd) {
            uint4 pk;
            pk.x = pack_bf16(v[q4 * 8 + 0] * inv, v[q4 * 8 + 1] * inv);
            pk.y = pack_bf16(v[q4 * 8 + 2] * inv, v[q4 * 8 + 3] * inv);
            pk.z = pack_bf16(v[q4 * 8 + 4] * inv, v[q4 * 8 + 5] * inv);
            pk.w = pack_bf16(v[q4 * 8 + 6] * inv, v[q4 * 8 + 7] * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + q4 * 8) = pk;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(COLS));
  }
}

template <int SPANS, int VSPANS>
int launch_latent(const __nv_bfloat16* q, const __nv_bfloat16* k_pool, __nv_bfloat16* out, const int* seq_q_start,
                  const int* seq_q_len, const int* seq_ctx_len, int table_row0, int n_seqs, int max_q_len, int n_tokens,
                  int n_heads, PagedView pv, int vd, float scale, int window, int min_len, int* status, cudaStream_t stream) {
  CUtensorMap mq, mk;
  int rc = tma_host::bf16_map(q, n_tokens, (long long)n_heads * pv.head_dim, BM, 64, &mq);
  if (rc) return rc;
  rc = tma_host::bf16_map(k_pool, pv.pool_rows, pv.head_dim, 16, 64, &mk);
  if (rc) return rc;
  static DeviceOnce once;
  const int dev_ = mf_current_device();
  if (dev_ < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev_]) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_latent_kernel<SPANS, VSPANS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)latent::smem(SPANS));
    if (e != cudaSuccess) return (int)e;
    once.done[dev_] = true;
  }
  dim3 grid(n_heads, (max_q_len + BM - 1) / BM, n_seqs);
  mf_count(MF_K_ATTN_PREFILL_TC);
  mf_count(MF_K_ATTN_PREFILL_LATENT);
  attn_prefill_latent_kernel<SPANS, VSPANS><<<grid, 192, latent::smem(SPANS), stream>>>(
      mq, mk, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, pv, n_heads, vd, scale * LOG2E, window, min_len, status);
  return (int)cudaGetLastError();
}

}  // namespace

// 1 (the default): portions of at least 128 tokens with head size 64 or 128 take the tcgen05
// kernel; 0: every shape takes the mma.sync kernel.  For tests and measurements.
MF_API int mf_set_prefill_tcgen05(int on) {
  g_prefill_tc = on ? 1 : 0;
  return 0;
}

// Arguments as launch_prefill of attention_prefill.cu plus the number of rows of q.  Returns
// MF_ERR_BAD_ARG when this kernel does not take the shape (the caller then uses the other one).
int launch_prefill_tc(const __nv_bfloat16* q, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool,
                      __nv_bfloat16* out, const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len,
                      int table_row0, int n_seqs, int max_q_len, int n_tokens, int n_heads, PagedView pv,
                      float scale, int window, int* status, cudaStream_t stream) {
  if (!g_prefill_tc || pv.page_size % 16 || max_q_len < BM || n_tokens <= 0 || pv.pool_rows <= 0) return MF_ERR_BAD_ARG;
  if ((((uintptr_t)q | (uintptr_t)out) & 15) != 0) return MF_ERR_BAD_ARG;
  if (pv.head_dim == 64)
    return launch_tc_ahead(q, k_pool, v_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs, max_q_len,
                           n_tokens, n_heads, pv, scale, window, status, stream);
  if (pv.head_dim == 128)
    return launch_pair<2, 2, true, false>(q, k_pool, v_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs,
                                          max_q_len, n_tokens, n_heads, pv, 128, scale, window, status, TcOptions{}, stream);
  return MF_ERR_BAD_ARG;
}

// Tokens of a tile of queries, and of the portions from which these kernels are taken.
int prefill_tc_rows() { return BM; }

// The same for attention with options; portions below `min_len` tokens are left out.  MF_ERR_BAD_ARG where the mma.sync kernel is the way: portions below 128 tokens, a soft
// cap, separate values of another size than head size 128, values inside the keys together with kept keys, a sink or
// a gate, a gate off its 16-byte boundary.
int launch_prefill_tc_ex(const __nv_bfloat16* q, const __nv_bfloat16* k_pool, const __nv_bfloat16* v_pool,
                         __nv_bfloat16* out, const int* seq_q_start, const int* seq_q_len, const int* seq_ctx_len,
                         int table_row0, int n_seqs, int max_q_len, int n_tokens, int n_heads, PagedView pv,
                         float scale, int window, const AttnOptions& opt, int min_len, int* status, cudaStream_t stream) {
  if (!g_prefill_tc || pv.page_size % 16 || max_q_len < BM || n_tokens <= 0 || pv.pool_rows <= 0 || opt.softcap > 0.f) return MF_ERR_BAD_ARG;
  if ((((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool) & 15) != 0 || (max_q_len + BM - 1) / BM > 65535) return MF_ERR_BAD_ARG;
  const int hd = pv.head_dim, vd = opt.vd;
  if (!opt.v_in_k) {
    if (hd != 128 || vd != 128 || ((uintptr_t)v_pool & 15) || (opt.gate && (((uintptr_t)opt.gate & 15) || opt.gate_ld % 8)))
      return MF_ERR_BAD_ARG;
    const TcOptions o{opt.keep_first, opt.sink, opt.gate, opt.gate_ld, min_len};
    return launch_pair<2, 2, true, true>(q, k_pool, v_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs,
                                         max_q_len, n_tokens, n_heads, pv, 128, scale, window, status, o, stream);
  }
  if (opt.sink || opt.gate || (window > 0 && opt.keep_first > 0) || hd <= 64 || vd % 16) return MF_ERR_BAD_ARG;
  const TcOptions o{0, nullptr, nullptr, 0, min_len};
  const int spans = (hd + 63) / 64, vspans = (vd + 63) / 64;
#define LATENT_GO(S, V)                                                                                                      \
  if (spans == S && vspans == V)                                                                                            \
  return launch_pair<S, V, false, true>(q, k_pool, k_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs,    \
                                        max_q_len, n_tokens, n_heads, pv, vd, scale, window, status, o, stream)
  LATENT_GO(2, 1);
  LATENT_GO(2, 2);
  LATENT_GO(3, 1);
  LATENT_GO(3, 2);
  LATENT_GO(3, 3);
  LATENT_GO(4, 2);
  LATENT_GO(4, 3);
  if (spans == 4 && vspans == 4)       // two chains' results do not fit in tensor memory beside their scores
    return launch_latent<4, 4>(q, k_pool, out, seq_q_start, seq_q_len, seq_ctx_len, table_row0, n_seqs, max_q_len, n_tokens,
                               n_heads, pv, vd, scale, window, min_len, status, stream);
#undef LATENT_GO
  return MF_ERR_BAD_ARG;
}
