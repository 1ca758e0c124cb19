// Retention over chunks of 64 tokens (see retention.cu for the rule itself).
//
// Per head, with the state S_0 before a chunk of n tokens (numbered from 0) and the head's decay g,
//
//   o_t = g^(t+1) S_0^T q_t + sum_(s <= t) g^(t-s) (q_t . k_s) v_s ,     S_n = g^n S_0 + sum_s g^(n-1-s) k_s v_s^T .
//
// The decay is one number, so chunks need nothing of one another but S_0:
//  * retention_local: what every chunk adds to the state, all chunks side by side;
//  * retention_carry: the states at the starts of the chunks, in place of those sums, and the sequence's last state;
//  * retention_chunk_out: the read-outs of all chunks side by side.
// Powers of the decay are worked out in double.  Values in 32 bits: IEEE 32-bit on the CUDA cores.  Values in bfloat16: on the tensor cores
// (mma.sync) with q, k, states and weights in three bfloat16 pieces that hold all 24 bits; of two such factors the six products of pieces
// down to 2^-16 of the leading one.  The unit cuts sums off where IEEE rounds, so 16 terms at a time are summed in it, the leading pieces (whose
// products have 16 bits) by themselves, and joined in IEEE 32-bit.
//
// Why: the recurrence token after token is serial (0.13 us a token), and its blocks, started early beside the tail of
// the kernel before them, stacked up on the few SMs that had room first.  1,777 tokens of 8 heads of 128 x 128, bfloat16 values: 244 ->
// 64 us on the CUDA cores (19 + 7 + 35; 850 us before when launches were queued back to back) -> 50 on the tensor cores (12 + 7 + 29 and the
// gaps between them), 2,048 of 16 heads 485 -> 120 -> 95, 300 tokens 37 -> 34; and a read-out is nearer to 64 bits (1.66e-7 of its norm, 1.81e-7 before, a
// state 1.78e-7, 1.85e-7).  On the CUDA cores the products hold about half of the FMA pipe's rate (counters: the FMA pipe 46 % busy,
// shared memory's 55 %), in one wave of blocks.  They run 8 x 8 results a thread (4 x 8 where the tile is smaller), because a lane
// gets four bytes a cycle from shared memory at most.  On the tensor cores 650 mma.sync a warp of the read-outs, 13 cycles each and
// scheduler in a loop of nothing else, are 60 % of the time of an SM that has two blocks; the rest is what cuts operands into pieces and waits for them
// (counters: tensor pipe 27 % busy, 36 where two blocks share an SM, issue slots 42 %).
#include "common.cuh"

namespace {
constexpr int L = 64;                    // tokens of a chunk
constexpr int LP = L + 4;                // a row of a transposed tile: rows of 16-byte pieces, neighbours in other banks

__device__ __forceinline__ bool find_chunk(int i, const int* __restrict__ q_len, int n_seqs, int& seq, int& chunk) {
  for (seq = 0; seq < n_seqs; seq++) {
    const int chunks = (q_len[seq] + L - 1) / L;
    if (i < chunks) {
      chunk = i;
      return true;
    }
    i -= chunks;
  }
  return false;
}

// g^n for 0 <= n <= L, g^0 = 1 (also of 0)
__device__ __forceinline__ float power(float g, int n) {
  double r = 1.0, b = g;
  for (int m = n; m; m >>= 1, b *= b)
    if (m & 1) r *= b;
  return (float)r;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// acc[i][j] += sum_k a[k][row i] b[k][column j] over K rows of two tiles in shared memory.  A thread's rows are four
// neighbours from `a` on and, for eight, four more `rstep` further; its columns likewise.  Sums of 16 products, then sums of
// those: chains as short as the ones of the recurrence's lanes.
template <int ROWS, int COLS>
__device__ __forceinline__ void tile_product(float (&acc)[ROWS][COLS], const float* a, int lda, int rstep, const float* b,
                                             int ldb, int cstep, int K) {
  for (int k0 = 0; k0 < K; k0 += 16) {
    float part[ROWS][COLS];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      float x[ROWS], y[COLS];
#pragma unroll
      for (int i = 0; i < ROWS; i += 4) *reinterpret_cast<float4*>(x + i) = load4(a + (k0 + k) * lda + i / 4 * rstep);
#pragma unroll
      for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(y + j) = load4(b + (k0 + k) * ldb + j / 4 * cstep);
#pragma unroll
      for (int i = 0; i < ROWS; i++)
#pragma unroll
        for (int j = 0; j < COLS; j++) part[i][j] = k == 0 ? x[i] * y[j] : fmaf(x[i], y[j], part[i][j]);
    }
#pragma unroll
    for (int i = 0; i < ROWS; i++)
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[i][j] += part[i][j];
  }
}

// ---------------------------------------------------------------------------- what a chunk adds to the state
// A block per (chunk, head), D V / 64 threads with 8 x 8 results each.
template <int D, int V>
__global__ void __launch_bounds__(D * V / 64)
retention_local_kernel(const float* __restrict__ qk, const float* __restrict__ v, long long v_ld,
                       const float* __restrict__ decay, const int* __restrict__ seq_q_start,
                       const int* __restrict__ seq_q_len, int n_seqs, float* __restrict__ states, int n_heads) {
  constexpr int THREADS = D * V / 64;
  extern __shared__ __align__(16) float sm[];
  float* ks = sm;                        // [L][D], times g^(n-1-s); rows from n on are zero
  float* vs = sm + L * D;                // [L][V]
  __shared__ float pw[L];
  int seq, chunk;
  if (!find_chunk(blockIdx.x, seq_q_len, n_seqs, seq, chunk)) return;
  const int h = blockIdx.y;
  const int n = min(L, seq_q_len[seq] - chunk * L);
  const long long t0 = seq_q_start[seq] + chunk * L;
  for (int i = threadIdx.x; i < L; i += THREADS) pw[i] = i < n ? power(decay[h], n - 1 - i) : 0.f;
  __syncthreads();
#pragma unroll
  for (int i = threadIdx.x; i < L * D / 4; i += THREADS) {
    const int s = i / (D / 4), c = i % (D / 4) * 4;
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s < n) {
      k = load4(qk + (t0 + s) * 2 * n_heads * D + (long long)(n_heads + h) * D + c);
      const float w = pw[s];
      k.x *= w; k.y *= w; k.z *= w; k.w *= w;
    }
    *reinterpret_cast<float4*>(ks + s * D + c) = k;
  }
#pragma unroll
  for (int i = threadIdx.x; i < L * V / 4; i += THREADS) {
    const int s = i / (V / 4), c = i % (V / 4) * 4;
    *reinterpret_cast<float4*>(vs + s * V + c) =
        s < n ? load4(v + (t0 + s) * v_ld + (long long)h * V + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  const int r = threadIdx.x / (V / 8) * 4, c = threadIdx.x % (V / 8) * 4;
  float acc[8][8] = {};
  tile_product<8, 8>(acc, ks + r, D, D / 2, vs + c, V, V / 2, (n + 15) / 16 * 16);
  float* out = states + ((long long)blockIdx.x * n_heads + h) * D * V;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    float* row = out + (r + (i & 3) + (i >> 2) * (D / 2)) * V + c;
    *reinterpret_cast<float4*>(row) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float4*>(row + V / 2) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
}

// ---------------------------------------------------------------------------- from chunk to chunk
// states [chunks][heads][D V]: a chunk's sum becomes the state it starts from; the slot gets the last one.
__global__ void __launch_bounds__(128)
retention_carry_kernel(float* __restrict__ states, const float* __restrict__ decay, float* __restrict__ state,
                       long long state_stride, const int* __restrict__ seq_q_len, const int* __restrict__ slots,
                       int n_heads, int size) {
  const int seq = blockIdx.x, h = blockIdx.y;
  const int e = (blockIdx.z * 128 + threadIdx.x) * 4;
  if (e >= size) return;
  const int n = seq_q_len[seq], chunks = (n + L - 1) / L;
  long long first = 0;
  for (int i = 0; i < seq; i++) first += (seq_q_len[i] + L - 1) / L;
  float* p = states + (first * n_heads + h) * size + e;
  const long long step = (long long)n_heads * size;
  float* own = state + (long long)slots[seq] * state_stride + (long long)h * size + e;
  const float g = power(decay[h], L), g_last = power(decay[h], n - (chunks - 1) * L);
  float4 s = load4(own);
  constexpr int AHEAD = 8;
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
    float4 a[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
      if (c0 + i < chunks) a[i] = load4(p + (c0 + i) * step);
#pragma unroll
    for (int i = 0; i < AHEAD; i++)
      if (c0 + i < chunks) {
        *reinterpret_cast<float4*>(p + (c0 + i) * step) = s;
        const float w = c0 + i == chunks - 1 ? g_last : g;
        s.x = fmaf(w, s.x, a[i].x);
        s.y = fmaf(w, s.y, a[i].y);
        s.z = fmaf(w, s.z, a[i].z);
        s.w = fmaf(w, s.w, a[i].w);
      }
  }
  *reinterpret_cast<float4*>(own) = s;
}

// ---------------------------------------------------------------------------- the read-outs
// A block of 2 V threads per (chunk, head): P = q k^T under the decays (written transposed), then S_0^T q and v^T P, 4 x 8
// results a thread.  q, k transposed in shared memory; k's room is v's and the state's (64 rows at a time) afterwards, so
// that two blocks share an SM.
template <int D, int V>
constexpr size_t chunk_out_smem() {
  const int b = D * LP > L * V ? D * LP : L * V;
  return (size_t)(D * LP + b + L * LP) * sizeof(float);
}

template <int D, int V>
__global__ void __launch_bounds__(2 * V, 2)
retention_chunk_out_kernel(const float* __restrict__ qk, const float* __restrict__ v, long long v_ld,
                           const float* __restrict__ decay, const int* __restrict__ seq_q_start,
                           const int* __restrict__ seq_q_len, int n_seqs, const float* __restrict__ states,
                           float* __restrict__ o_out, int n_heads) {
  constexpr int THREADS = 2 * V;
  constexpr int PC = L * L / 4 / THREADS;          // columns of a thread's tile of P: 4 at 256 threads, 8 at 128
  extern __shared__ __align__(16) float sm[];
  float* qt = sm;                        // [D][LP]
  float* bt = sm + D * LP;               // k transposed [D][LP]; then the state [64][V] and v [L][V]
  float* pt = bt + (D * LP > L * V ? D * LP : L * V);          // [L][LP]: P transposed
  __shared__ float pw[L + 1];
  int seq, chunk;
  if (!find_chunk(blockIdx.x, seq_q_len, n_seqs, seq, chunk)) return;
  const int h = blockIdx.y, tid = threadIdx.x;
  const int n = min(L, seq_q_len[seq] - chunk * L);
  const long long t0 = seq_q_start[seq] + chunk * L;
  for (int i = tid; i <= L; i += THREADS) pw[i] = power(decay[h], i);
  // a lane takes eight channels (a sector) of a token, neighbouring lanes neighbouring tokens
#pragma unroll 4
  for (int i = tid; i < 2 * L * (D / 8); i += THREADS) {
    const int t = i % L, rest = i / L, which = rest / (D / 8), c = rest % (D / 8) * 8;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    if (t < n) {
      const float* p = qk + (t0 + t) * 2 * n_heads * D + (long long)(which * n_heads + h) * D + c;
      x = load4(p);
      y = load4(p + 4);
    }
    float* dst = (which ? bt : qt) + c * LP + t;
    dst[0] = x.x; dst[LP] = x.y; dst[2 * LP] = x.z; dst[3 * LP] = x.w;
    dst[4 * LP] = y.x; dst[5 * LP] = y.y; dst[6 * LP] = y.z; dst[7 * LP] = y.w;
  }
  __syncthreads();
  {
    const int r = tid / (L / PC) * 4, c = tid % (L / PC) * 4;
    float p[4][PC] = {};
    tile_product<4, PC>(p, qt + r, LP, 0, bt + c, LP, 32, D);
#pragma unroll
    for (int j = 0; j < PC; j++) {
      const int s = c + (j & 3) + (j >> 2) * 32;
      float w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) w[i] = r + i >= s ? p[i][j] * pw[r + i - s] : 0.f;
      *reinterpret_cast<float4*>(pt + s * LP + r) = make_float4(w[0], w[1], w[2], w[3]);
    }
  }
  const int r = tid / (V / 8) * 4, c = tid % (V / 8) * 4;
  float acc[4][8] = {};
  const float* from = states + ((long long)blockIdx.x * n_heads + h) * D * V;
#pragma unroll
  for (int d0 = 0; d0 < D; d0 += 64) {
    __syncthreads();
#pragma unroll
    for (int i = tid; i < 64 * V / 4; i += THREADS)
      reinterpret_cast<float4*>(bt)[i] = load4(from + (long long)d0 * V + i * 4);
    __syncthreads();
    tile_product<4, 8>(acc, qt + d0 * LP + r, LP, 0, bt + c, V, V / 2, 64);
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float w = pw[r + i + 1];
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] *= w;
  }
  __syncthreads();
#pragma unroll
  for (int i = tid; i < L * V / 4; i += THREADS) {
    const int s = i / (V / 4), cc = i % (V / 4) * 4;
    reinterpret_cast<float4*>(bt)[i] =
        s < n ? load4(v + (t0 + s) * v_ld + (long long)h * V + cc) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  // keys behind a row's own group of 16 do not count; of that group each row takes its own tokens alone: a weight of zero would
  // let a value that is not finite into the tokens before it
  const int own = r / 16 * 16;
  tile_product<4, 8>(acc, pt + r, LP, 0, bt + c, V, V / 2, min((n + 15) / 16 * 16, own));
  if (own < n) {
    float part[4][8] = {};
#pragma unroll
    for (int k = 0; k < 16; k++) {
      float x[4], y[8];
      *reinterpret_cast<float4*>(x) = load4(pt + (own + k) * LP + r);
      *reinterpret_cast<float4*>(y) = load4(bt + (own + k) * V + c);
      *reinterpret_cast<float4*>(y + 4) = load4(bt + (own + k) * V + c + V / 2);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (own + k <= r + i) {
#pragma unroll
          for (int j = 0; j < 8; j++) part[i][j] = fmaf(x[i], y[j], part[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[i][j] += part[i][j];
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int t = r + i;
    if (t >= n) continue;
    float* row = o_out + (t0 + t) * n_heads * V + (long long)h * V + c;
    *reinterpret_cast<float4*>(row) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float4*>(row + V / 2) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
}

// ---------------------------------------------------------------------------- the same on the tensor cores
// two 32-bit numbers as three pairs of bfloat16 whose sums they are.  Of what is infinite, or larger than bfloat16's largest, the first is an
// infinity and the others are no numbers; a bfloat16 infinity meets pieces of either sign, or zeros.  Every product such a number is in
// comes out as something that is not finite, so the kernels below work out those results again in IEEE 32-bit, and no others.
__device__ __forceinline__ void pieces(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    p[i] = *reinterpret_cast<const uint32_t*>(&b);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 rows x 16 terms of a 32-bit matrix as A operands of its pieces: `at(row, term)` gives two neighbouring terms
template <typename At>
__device__ __forceinline__ void a_pieces(uint32_t (&a)[3][4], At at) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 x = at((i & 1) * 8, (i >> 1) * 8);
    uint32_t p[3];
    pieces(x.x, x.y, p);
    a[0][i] = p[0], a[1][i] = p[1], a[2][i] = p[2];
  }
}
// sum += A B over 16 terms, B 16 terms x 8 columns in three pieces
__device__ __forceinline__ void add_product(float (&sum)[4], const uint32_t (&a)[3][4], const uint32_t (&b0)[3], const uint32_t (&b1)[3]) {
  float t[4] = {}, rest[4] = {};
  mma(t, a[0], b0[0], b1[0]);
  mma(rest, a[2], b0[0], b1[0]);
  mma(rest, a[0], b0[2], b1[2]);
  mma(rest, a[1], b0[1], b1[1]);
  mma(rest, a[1], b0[0], b1[0]);
  mma(rest, a[0], b0[1], b1[1]);
#pragma unroll
  for (int e = 0; e < 4; e++) sum[e] += t[e] + rest[e];
}
// the same where B is bfloat16 as it is
__device__ __forceinline__ void add_product(float (&sum)[4], const uint32_t (&a)[3][4], uint32_t b0, uint32_t b1) {
  float t[4] = {}, rest[4] = {};
  mma(t, a[0], b0, b1);
  mma(rest, a[2], b0, b1);
  mma(rest, a[1], b0, b1);
#pragma unroll
  for (int e = 0; e < 4; e++) sum[e] += t[e] + rest[e];
}
// values of 16 tokens from `row` on (rows of `ld`), 16 columns: the B operands of two products of eight columns
__device__ __forceinline__ void value_operands(uint32_t (&b)[4], const __nv_bfloat16* row, int ld, int lane) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(row + (lane & 15) * ld + (lane >> 4) * 8);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(at));
}
__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) <= 3.402823466e38f); }
template <int V, int THREADS>
__device__ __forceinline__ void copy_values(__nv_bfloat16* vs, const __nv_bfloat16* v, long long v_ld, int n) {
#pragma unroll 4
  for (int i = threadIdx.x; i < L * V / 4; i += THREADS) {
    const int s = i / (V / 4), c = i % (V / 4) * 4;
    *reinterpret_cast<uint2*>(vs + s * (V + 8) + c) = s < n ? *reinterpret_cast<const uint2*>(v + s * v_ld + c) : make_uint2(0, 0);
  }
}

// A block per (chunk, head), a warp per 16 channels of the keys, which are the rows of the product.  1,777 tokens of 8 heads of 128 x 128:
// 20 us on the CUDA cores (half of their rate).
template <int D, int V>
constexpr size_t local_mma_smem() { return (size_t)L * (D + 4) * 4 + (size_t)L * (V + 8) * 2; }

// a thread's results that are not finite: of a step of eight columns two neighbours, and those eight rows further
template <int D, int V>
__device__ __noinline__ void local_again(float* out, const float* ks, const __nv_bfloat16* vs, int n) {
#pragma unroll 1
  for (int i = 0; i < V / 2; i++) {
    const int row = (i & 2) * 4, col = i / 4 * 8 + (i & 1);
    if (!not_finite(out[row * V + col])) continue;
    float x = 0.f;
#pragma unroll 1
    for (int s = 0; s < n; s++) x = fmaf(ks[s * (D + 4) + row], __bfloat162float(vs[s * (V + 8) + col]), x);
    out[row * V + col] = x;
  }
}

template <int D, int V>
__global__ void __launch_bounds__(2 * D, 2)
retention_local_mma_kernel(const float* __restrict__ qk, const __nv_bfloat16* __restrict__ v, long long v_ld, const float* __restrict__ decay,
                           const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int n_seqs, float* __restrict__ states,
                           int n_heads) {
  constexpr int THREADS = 2 * D, K_LD = D + 4;
  extern __shared__ __align__(16) float sm[];
  float* ks = sm;                                                           // [L][K_LD], times g^(n-1-s); rows from n on are zero
  __nv_bfloat16* vs = reinterpret_cast<__nv_bfloat16*>(sm + L * K_LD);      // [L][V + 8]
  __shared__ float pw[L];
  int seq, chunk;
  if (!find_chunk(blockIdx.x, seq_q_len, n_seqs, seq, chunk)) return;
  const int h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = lane >> 2, c2 = (lane & 3) * 2;
  const int n = min(L, seq_q_len[seq] - chunk * L);
  const long long t0 = seq_q_start[seq] + chunk * L;
  for (int i = threadIdx.x; i < L; i += THREADS) pw[i] = i < n ? power(decay[h], n - 1 - i) : 0.f;
  copy_values<V, THREADS>(vs, v + t0 * v_ld + (long long)h * V, v_ld, n);
  __syncthreads();
#pragma unroll 4
  for (int i = threadIdx.x; i < L * D / 4; i += THREADS) {
    const int s = i / (D / 4), c = i % (D / 4) * 4;
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s < n) {
      k = load4(qk + (t0 + s) * 2 * n_heads * D + (long long)(n_heads + h) * D + c);
      const float w = pw[s];
      k.x *= w; k.y *= w; k.z *= w; k.w *= w;
    }
    *reinterpret_cast<float4*>(ks + s * K_LD + c) = k;
  }
  __syncthreads();
  float acc[V / 8][4] = {};
  for (int s0 = 0; s0 < n; s0 += 16) {
    uint32_t a[3][4];
    a_pieces(a, [&](int row, int term) {
      const float* at = ks + (s0 + term + c2) * K_LD + warp * 16 + r0 + row;
      return make_float2(at[0], at[K_LD]);
    });
#pragma unroll
    for (int j = 0; j < V / 8; j += 2) {
      uint32_t b[4];
      value_operands(b, vs + s0 * (V + 8) + j * 8, V + 8, lane);
      add_product(acc[j], a, b[0], b[1]);
      add_product(acc[j + 1], a, b[2], b[3]);
    }
  }
  float* out = states + ((long long)blockIdx.x * n_heads + h) * D * V + (warp * 16 + r0) * V + c2;
  bool again = false;
#pragma unroll
  for (int j = 0; j < V / 8; j++) {
    *reinterpret_cast<float2*>(out + j * 8) = make_float2(acc[j][0], acc[j][1]);
    *reinterpret_cast<float2*>(out + 8 * V + j * 8) = make_float2(acc[j][2], acc[j][3]);
#pragma unroll
    for (int e = 0; e < 4; e++) again |= not_finite(acc[j][e]);
  }
  if (again) local_again<D, V>(out, ks + warp * 16 + r0, vs + c2, n);
}

// A block of 2 V threads per (chunk, head): P = q k^T under the decays, then q S_0 and P v; a warp has 16 tokens and 64 columns.  q, k, the
// state (64 rows at a time) and P stand in shared memory in 32 bits and are cut into pieces on their way into registers: 22 instructions
// for the operand of six products that take 78 cycles.  1,777 tokens of 8 heads of 128 x 128: 35 us on the CUDA cores.
template <int D, int V>
constexpr size_t out_mma_smem() {
  const int b = D + 8 > V + 4 ? D + 8 : V + 4;
  return (size_t)L * (D + 8 + b + L + 8) * 4 + (size_t)L * (V + 8) * 2;
}

// A chunk's weights and results that are not finite, by the whole block; behind the kernel's end, where nothing of it is held in registers
// (a look at the weights where they are made took 2 us of 50).  `qk`, `state`, `out`: the chunk's and head's first.
template <int D, int V>
__device__ __noinline__ void read_again(const float* qk, long long qk_ld, int k_off, const float* state, float* out, long long out_ld, const float* qs,
                                        float* ps, const float* pw, const __nv_bfloat16* vs, int n) {
  for (int i = threadIdx.x; i < n * L; i += 2 * V) {
    const int t = i / L, key = i % L;
    if (key > t || !not_finite(ps[t * (L + 8) + key])) continue;
    float x = 0.f;
#pragma unroll 1
    for (int d = 0; d < D; d++) x = fmaf(qs[t * (D + 8) + d], qk[key * qk_ld + k_off + d], x);
    ps[t * (L + 8) + key] = x * pw[t - key];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * V; i += 2 * V) {
    const int t = i / V, c = i % V;
    float* const to = out + t * out_ld + c;
    if (!not_finite(*to)) continue;
    float x = 0.f;
#pragma unroll 1
    for (int d = 0; d < D; d++) x = fmaf(qs[t * (D + 8) + d], state[d * V + c], x);
    x *= pw[t + 1];
#pragma unroll 1
    for (int s = 0; s <= t; s++) x = fmaf(ps[t * (L + 8) + s], __bfloat162float(vs[s * (V + 8) + c]), x);
    *to = x;
  }
}

template <int D, int V>
__global__ void __launch_bounds__(2 * V, 2)
retention_out_mma_kernel(const float* __restrict__ qk, const __nv_bfloat16* __restrict__ v, long long v_ld, const float* __restrict__ decay,
                         const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int n_seqs, const float* __restrict__ states,
                         float* __restrict__ o_out, int n_heads) {
  constexpr int THREADS = 2 * V, Q_LD = D + 8, S_LD = V + 4, P_LD = L + 8, B = Q_LD > S_LD ? Q_LD : S_LD, HALVES = V / 64;
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                        // [L][Q_LD]
  float* bs = qs + L * Q_LD;             // k [L][Q_LD]; then 64 rows of the state [64][S_LD]
  float* ps = bs + L * B;                // [L][P_LD]
  __nv_bfloat16* vs = reinterpret_cast<__nv_bfloat16*>(ps + L * P_LD);      // [L][V + 8]
  __shared__ float pw[L + 1];
  int seq, chunk;
  if (!find_chunk(blockIdx.x, seq_q_len, n_seqs, seq, chunk)) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r0 = lane >> 2, c2 = (lane & 3) * 2;
  const int half = warp >> 2, group = half ? 3 - (warp & 3) : warp & 3;     // 16 tokens; a scheduler gets early and late ones
  const int n = min(L, seq_q_len[seq] - chunk * L), row = group * 16 + r0;
  const long long t0 = seq_q_start[seq] + chunk * L;
  for (int i = tid; i <= L; i += THREADS) pw[i] = power(decay[h], i);
#pragma unroll 8
  for (int i = tid; i < 2 * L * (D / 4); i += THREADS) {
    const int which = i / (L * (D / 4)), t = i / (D / 4) % L, c = i % (D / 4) * 4;
    *reinterpret_cast<float4*>((which ? bs : qs) + t * Q_LD + c) =
        t < n ? load4(qk + (t0 + t) * 2 * n_heads * D + (long long)(which * n_heads + h) * D + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  copy_values<V, THREADS>(vs, v + t0 * v_ld + (long long)h * V, v_ld, n);
  // the next 64 rows of the state are on their way while something else is worked on
  const float* from = states + ((long long)blockIdx.x * n_heads + h) * D * V;
  float4 ahead[8];
  auto fetch = [&](int d0) {
#pragma unroll
    for (int i = 0; i < 8; i++) ahead[i] = load4(from + (long long)d0 * V + (tid + i * THREADS) * 4);
  };
  fetch(0);
  __syncthreads();
  auto queries = [&](uint32_t (&a)[3][4], int d) {
    a_pieces(a, [&](int r, int term) { return *reinterpret_cast<const float2*>(qs + (row + r) * Q_LD + d + term + c2); });
  };
  {
    constexpr int NT = 8 / HALVES;                                           // columns of eight keys
    float p[NT][4] = {};
    const int key0 = half * NT * 8;
#pragma unroll 2
    for (int d = 0; d < D; d += 16) {
      uint32_t a[3][4];
      queries(a, d);
#pragma unroll
      for (int j = 0; j < NT; j++) {
        if (key0 + j * 8 > group * 16 + 15) break;
        const float* at = bs + (key0 + j * 8 + r0) * Q_LD + d + c2;
        const float2 x = *reinterpret_cast<const float2*>(at), y = *reinterpret_cast<const float2*>(at + 8);
        uint32_t b0[3], b1[3];
        pieces(x.x, x.y, b0);
        pieces(y.x, y.y, b1);
        add_product(p[j], a, b0, b1);
      }
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
      const int key = key0 + j * 8 + c2;
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int t = row + e * 4;
        *reinterpret_cast<float2*>(ps + t * P_LD + key) =
            make_float2(t >= key ? p[j][e] * pw[t - key] : 0.f, t >= key + 1 ? p[j][e + 1] * pw[t - key - 1] : 0.f);
      }
    }
  }
  float acc[8][4] = {};
#pragma unroll 1
  for (int d0 = 0; d0 < D; d0 += 64) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int at = (tid + i * THREADS) * 4;
      *reinterpret_cast<float4*>(bs + at / V * S_LD + at % V) = ahead[i];
    }
    if (d0 + 64 < D) fetch(d0 + 64);
    __syncthreads();
#pragma unroll 1
    for (int d = 0; d < 64; d += 16) {
      uint32_t a[3][4];
      queries(a, d0 + d);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float* at = bs + (d + c2) * S_LD + half * 64 + j * 8 + r0;
        uint32_t b0[3], b1[3];
        pieces(at[0], at[S_LD], b0);
        pieces(at[8 * S_LD], at[9 * S_LD], b1);
        add_product(acc[j], a, b0, b1);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[j][e] *= pw[row + (e >> 1) * 8 + 1];
  // keys of the groups of 16 before a row's own; of its own group each row takes its own tokens alone: a weight of zero would let a value
  // that is not finite into the tokens before it
  const __nv_bfloat16* vh = vs + half * 64;
#pragma unroll 1
  for (int g = 0; g < group && g * 16 < n; g++) {
    uint32_t a[3][4];
    a_pieces(a, [&](int r, int term) { return *reinterpret_cast<const float2*>(ps + (row + r) * P_LD + g * 16 + term + c2); });
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      uint32_t b[4];
      value_operands(b, vh + g * 16 * (V + 8) + j * 8, V + 8, lane);
      add_product(acc[j], a, b[0], b[1]);
      add_product(acc[j + 1], a, b[2], b[3]);
    }
  }
  if (group * 16 < n) {
    float part[8][4] = {};
#pragma unroll 2
    for (int k = 0; k < 16; k++) {
      const int key = group * 16 + k;
      const float w0 = ps[row * P_LD + key], w1 = ps[(row + 8) * P_LD + key];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint32_t u = *reinterpret_cast<const uint32_t*>(vh + key * (V + 8) + j * 8 + c2);
        const float x = __uint_as_float(u << 16), y = __uint_as_float(u & 0xffff0000u);
        if (key <= row) part[j][0] = fmaf(w0, x, part[j][0]), part[j][1] = fmaf(w0, y, part[j][1]);
        if (key <= row + 8) part[j][2] = fmaf(w1, x, part[j][2]), part[j][3] = fmaf(w1, y, part[j][3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[j][e] += part[j][e];
  }
  bool again = false;
#pragma unroll
  for (int e = 0; e < 4; e += 2) {
    const int t = row + e * 4;
    if (t >= n) continue;
    float* to = o_out + (t0 + t) * n_heads * V + (long long)h * V + half * 64 + c2;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      *reinterpret_cast<float2*>(to + j * 8) = make_float2(acc[j][e], acc[j][e + 1]);
      again |= not_finite(acc[j][e]) | not_finite(acc[j][e + 1]);
    }
  }
  if (__syncthreads_or(again))
    read_again<D, V>(qk + t0 * 2 * n_heads * D + (long long)h * D, 2ll * n_heads * D, n_heads * D, from, o_out + t0 * n_heads * V + (long long)h * V,
                     (long long)n_heads * V, qs, ps, pw, vs, n);
}

template <typename T, int D, int V>
int launch(const float* qk, const T* v, long long v_ld, const float* decay, float* state, long long state_stride,
           const int* seq_q_start, const int* seq_q_len, const int* slots, float* o_out, int n_seqs, int n_chunks,
           int n_heads, float* scratch, cudaStream_t stream) {
  constexpr bool MMA = sizeof(T) == 2;
  constexpr size_t local_smem = MMA ? local_mma_smem<D, V>() : (size_t)L * (D + V) * sizeof(float);
  constexpr size_t out_smem = MMA ? out_mma_smem<D, V>() : chunk_out_smem<D, V>();
  const auto local = [] {
    if constexpr (MMA) return retention_local_mma_kernel<D, V>;
    else return retention_local_kernel<D, V>;
  }();
  const auto read = [] {
    if constexpr (MMA) return retention_out_mma_kernel<D, V>;
    else return retention_chunk_out_kernel<D, V>;
  }();
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(local, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)local_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(read, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  local<<<dim3(n_chunks, n_heads), MMA ? 2 * D : D * V / 64, local_smem, stream>>>(qk, v, v_ld, decay, seq_q_start, seq_q_len, n_seqs, scratch,
                                                                                 n_heads);
  retention_carry_kernel<<<dim3(n_seqs, n_heads, D * V / 512), 128, 0, stream>>>(scratch, decay, state, state_stride,
                                                                                 seq_q_len, slots, n_heads, D * V);
  read<<<dim3(n_chunks, n_heads), 2 * V, out_smem, stream>>>(qk, v, v_ld, decay, seq_q_start, seq_q_len, n_seqs, scratch, o_out, n_heads);
  return (int)cudaGetLastError();
}
}  // namespace

// Heads of 64 or 128 channels with values of 64 or 128, rows of whole 16-byte pieces (8 for bfloat16 values).
MF_API int mf_retention_chunked_ok(int dim, int vdim, long long v_ld) {
  return (dim == 64 || dim == 128) && (vdim == 64 || vdim == 128) && v_ld % 4 == 0;
}

// Arguments as for mf_retention_recurrence, with one partial read-out.  `n_chunks`: the sum of ceil(q_len / 64) over the
// sequences; `scratch`: n_chunks * n_heads * dim * vdim floats.
MF_API int mf_retention_chunked(const float* qk, const void* v, int v_dtype, long long v_ld, const float* decay,
                                float* state, long long state_stride, const int* seq_q_start, const int* seq_q_len,
                                const int* slots, float* o_out, int n_seqs, int n_chunks, int n_heads, int dim, int vdim,
                                float* scratch, cudaStream_t stream) {
  if (n_seqs <= 0 || n_chunks <= 0) return 0;
  const int piece = v_dtype == MF_F32 ? 16 : 8;
  if (!mf_retention_chunked_ok(dim, vdim, v_ld) || n_heads <= 0 || n_heads > 65535 || ((uintptr_t)qk & 15) ||
      ((uintptr_t)v % piece) || ((uintptr_t)scratch & 15) || ((uintptr_t)o_out & 15) || ((uintptr_t)state & 15) ||
      state_stride % 4)
    return MF_ERR_BAD_ARG;
  mf_count(MF_K_RETENTION_CHUNKED);
#define RC_GO(T, D, V)                                                                                              \
  return launch<T, D, V>(qk, (const T*)v, v_ld, decay, state, state_stride, seq_q_start, seq_q_len, slots, o_out,   \
                         n_seqs, n_chunks, n_heads, scratch, stream)
#define RC_SIZES(T)                              \
  if (dim == 64 && vdim == 64) RC_GO(T, 64, 64);   \
  if (dim == 64) RC_GO(T, 64, 128);                \
  if (vdim == 64) RC_GO(T, 128, 64);               \
  RC_GO(T, 128, 128)
  if (v_dtype == MF_F32) { RC_SIZES(float); }
  if (v_dtype == MF_BF16) { RC_SIZES(__nv_bfloat16); }
#undef RC_SIZES
#undef RC_GO
  return MF_ERR_BAD_DTYPE;
}
