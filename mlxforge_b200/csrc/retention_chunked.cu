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
// All of it is IEEE 32-bit on the CUDA cores (q and k are 32-bit: rounding them to a tensor-core type would lose what the
// rotation kept); powers of the decay are worked out in double.
//
// Why: the recurrence token after token is serial (0.13 us a token), and its blocks, started early beside the tail of
// the kernel before them, stacked up on the few SMs that had room first.  1,777 tokens of 8 heads of 128 x 128: 244 ->
// 64 us (19 + 7 + 35; 850 us before when launches were queued back to back), 2,048 of 16 heads: 485 -> 120 us.  The
// products hold about half of the FMA pipe's rate (counters: the FMA pipe 46 % busy, shared memory's 55 %), in one wave of blocks.
// They run 8 x 8 results a thread (4 x 8 where the tile is smaller), because a lane gets four bytes a cycle from shared
// memory at most.
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
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

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
template <typename T, int D, int V>
__global__ void __launch_bounds__(D * V / 64)
retention_local_kernel(const float* __restrict__ qk, const T* __restrict__ v, long long v_ld,
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

template <typename T, int D, int V>
__global__ void __launch_bounds__(2 * V, 2)
retention_chunk_out_kernel(const float* __restrict__ qk, const T* __restrict__ v, long long v_ld,
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

template <typename T, int D, int V>
int launch(const float* qk, const T* v, long long v_ld, const float* decay, float* state, long long state_stride,
           const int* seq_q_start, const int* seq_q_len, const int* slots, float* o_out, int n_seqs, int n_chunks,
           int n_heads, float* scratch, cudaStream_t stream) {
  constexpr size_t local_smem = (size_t)L * (D + V) * sizeof(float), out_smem = chunk_out_smem<D, V>();
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(retention_local_kernel<T, D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)local_smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(retention_chunk_out_kernel<T, D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  retention_local_kernel<T, D, V><<<dim3(n_chunks, n_heads), D * V / 64, local_smem, stream>>>(
      qk, v, v_ld, decay, seq_q_start, seq_q_len, n_seqs, scratch, n_heads);
  retention_carry_kernel<<<dim3(n_seqs, n_heads, D * V / 512), 128, 0, stream>>>(scratch, decay, state, state_stride,
                                                                                 seq_q_len, slots, n_heads, D * V);
  retention_chunk_out_kernel<T, D, V><<<dim3(n_chunks, n_heads), 2 * V, out_smem, stream>>>(
      qk, v, v_ld, decay, seq_q_start, seq_q_len, n_seqs, scratch, o_out, n_heads);
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
