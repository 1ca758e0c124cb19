// Retention: linear attention with a fixed decay per head and no softmax.  Per head, with a
// 32-bit state S [dim, vdim] per request that starts at zero:
//
//     S_t = decay_h S_(t-1) + k_t v_t^T ,     o_t = S_t^T q_t
//
// q and k are rotated by position (half-split pairs over the first `rot` channels), k is then
// multiplied by `k_scale`; each head's o_t is divided by its root mean square (no weight),
// multiplied by silu(gate) and handed to the output projection.
//
//  * retention_prepare: one block per token; rotation and key scaling into 32-bit [T, 2 heads dim].
//  * retention_recurrence: every column of S is independent, so the recurrence is parallel over
//    (sequence, head, column) and serial in time only.  Eight lanes share a column and hold
//    dim/8 of its rows in registers; q and k of the coming tokens are staged in shared memory,
//    eight tokens at a time.  A step continues from the slot's state, and which kernel takes a
//    sequence is a matter of its own portion: one token, token after token, or chunks of 64
//    (retention_chunked.cu).  The three add a read-out in other orders, so another cut of a prompt moves
//    it within 32-bit rounding; what else is in the step does not.
//  * retention_output: per token and head the read-out (summed over the row groups that a staged
//    launch spreads a head's state over) over its root mean square, times silu(gate).
#include "rotary.cuh"

namespace {
constexpr int RT_LANES = 8;                 // lanes that share one column of S
constexpr int RT_COLS = 16;                 // columns per block
constexpr int RT_THREADS = RT_LANES * RT_COLS;
constexpr int RT_CHUNK = 8;                 // tokens staged at a time
}  // namespace

// act 1: SiLU of every query and key channel before anything else.  v_out (optional): the row's `nv`
// channels from column `v_off` on, through the same activation, in 32-bit [T, nv].
template <typename T>
__global__ void retention_prepare_kernel(const T* proj, int ld, int n_heads, int dim, int rot,
                                         float k_scale, const int* positions,
                                         const float* __restrict__ inv_f, const double* __restrict__ inv_d,
                                         float* __restrict__ qk, int act, float* __restrict__ v_out, int v_off, int nv) {
  extern __shared__ float cs[];            // [half] cos, [half] sin
  pdl_launch();
  const int t = blockIdx.x;
  const int pos = positions[t];
  const int half = rot >> 1;
  for (int j = threadIdx.x; j < half; j += blockDim.x) rotary_cs(pos, j, inv_f, inv_d, cs[j], cs[half + j]);
  __syncthreads();
  pdl_wait();
  const T* row = proj + (long long)t * ld;
  float* out = qk + (long long)t * 2 * n_heads * dim;
  const int per_head = dim - half;
  auto rd = [&](const T* p) {
    const float x = to_f32<T>(*p);
    return act ? x / (1.0f + expf(-x)) : x;
  };
  for (int idx = threadIdx.x; idx < 2 * n_heads * per_head; idx += blockDim.x) {
    const int h = idx / per_head, j = idx - h * per_head;       // heads 0..n-1: queries, n..2n-1: keys
    const T* src = row + (long long)h * dim;
    float* dst = out + (long long)h * dim;
    const float f = h >= n_heads ? k_scale : 1.0f;
    if (j < half) {
      const float c = cs[j], s = cs[half + j];
      const float u = rd(src + j), v = rd(src + j + half);
      dst[j] = (u * c - v * s) * f;
      dst[j + half] = (v * c + u * s) * f;
    } else {
      const int ch = rot + (j - half);
      dst[ch] = rd(src + ch) * f;
    }
  }
  if (v_out)
    for (int i = threadIdx.x; i < nv; i += blockDim.x) v_out[(long long)t * nv + i] = rd(row + v_off + i);
}

// The same for bfloat16 rows in pieces of eight channels and of the eight they pair with (head size and half of the rotated channels
// multiples of 8, 16-byte aligned rows, no v_out), TOK tokens a block (mf_store_tokens), the angles of all of them side by side.
// 1,777 tokens of 8 heads of 128, half of the channels turned (22 MB, in L2): 10.3 us with a channel a thread, 5.5 here; all turned 10.6 and 7.6.
template <int TOK, int U>
__global__ void __launch_bounds__(256)
retention_prepare_vec_kernel(const __nv_bfloat16* proj, int ld, int n_heads, int dim, int rot, int T, float k_scale,
                             const int* positions, const float* __restrict__ inv_f,
                             const double* __restrict__ inv_d, float* __restrict__ qk, int act) {
  extern __shared__ float cs[];            // [TOK][half] cos, then sin
  pdl_launch();
  const int t0 = blockIdx.x * TOK, nt = TOK == 1 ? 1 : min(TOK, T - t0), half = rot >> 1;
  for (int i = threadIdx.x; i < nt * half; i += 256) {
    const int t = TOK == 1 ? 0 : i / half, j = i - t * half;
    rotary_cs(positions[t0 + t], j, inv_f, inv_d, cs[i], cs[TOK * half + i]);
  }
  __syncthreads();
  pdl_wait();
  auto unpack = [&](const uint4 u, float (&x)[8]) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 f = __bfloat1622float2(p[e]);
      x[2 * e] = act ? f.x / (1.0f + expf(-f.x)) : f.x;
      x[2 * e + 1] = act ? f.y / (1.0f + expf(-f.y)) : f.y;
    }
  };
  auto put = [](float* p, const float (&x)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(x[4], x[5], x[6], x[7]);
  };
  const int turned = half >> 3, per_head = turned + ((dim - rot) >> 3), per_token = 2 * n_heads * per_head;
  // U pieces a thread are on their way before the first is stored
  for (int i0 = threadIdx.x; i0 < nt * per_token; i0 += U * 256) {
    uint4 in[U], in2[U];
#pragma unroll
    for (int w = 0; w < U; w++) {
      const int i = i0 + w * 256, t = TOK == 1 ? 0 : i / per_token, rest = i - t * per_token;
      const int h = rest / per_head, c = rest - h * per_head;
      if (i >= nt * per_token) continue;
      const __nv_bfloat16* src =
          proj + (long long)(t0 + t) * ld + (long long)h * dim + (c < turned ? c * 8 : rot + (c - turned) * 8);
      in[w] = *reinterpret_cast<const uint4*>(src);
      if (c < turned) in2[w] = *reinterpret_cast<const uint4*>(src + half);
    }
#pragma unroll
    for (int w = 0; w < U; w++) {
      const int i = i0 + w * 256, t = TOK == 1 ? 0 : i / per_token, rest = i - t * per_token;
      const int h = rest / per_head, c = rest - h * per_head;
      if (i >= nt * per_token) continue;
      float* dst = qk + ((long long)(t0 + t) * 2 * n_heads + h) * dim;      // heads 0..n-1: queries, n..2n-1: keys
      const float f = h >= n_heads ? k_scale : 1.0f;
      float u[8], v[8];
      if (c < turned) {
        const int j = c * 8;
        unpack(in[w], u);
        unpack(in2[w], v);
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const float co = cs[t * half + j + e], si = cs[(TOK + t) * half + j + e];
          const float a = (u[e] * co - v[e] * si) * f, b = (v[e] * co + u[e] * si) * f;
          u[e] = a;
          v[e] = b;
        }
        put(dst + j, u);
        put(dst + j + half, v);
      } else {
        const int ch = rot + (c - turned) * 8;
        unpack(in[w], u);
#pragma unroll
        for (int e = 0; e < 8; e++) u[e] *= f;
        put(dst + ch, u);
      }
    }
  }
}

MF_API int mf_retention_prepare(const void* proj, int dtype, int T, int ld, int n_heads, int dim, int rot,
                                float k_scale, const int* positions, const float* inv_f, const double* inv_d,
                                float* qk, int act, float* v_out, int v_off, int nv, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (rot < 0 || rot > dim || (rot & 1) || (rot > 0 && !inv_f && !inv_d)) return MF_ERR_BAD_ARG;
  const size_t smem = (size_t)(rot > 0 ? rot : 1) * sizeof(float);
  mf_count(MF_K_RETENTION_PREPARE);
  if (dtype == MF_BF16 && !v_out && dim % 8 == 0 && rot % 16 == 0 && ld % 8 == 0 && 4 * smem <= 48 * 1024 &&
      !(((uintptr_t)proj | (uintptr_t)qk) & 15)) {
    // a piece here is two loads and four stores: four tokens a block from the first size on up to 128 of them (1,777 tokens of 8 heads of 128,
    // all channels turned, 8.3 / 7.6 us with one / four; 4 heads 6.2 / 5.3)
    if (mf_store_tokens(T, 2 * n_heads * ((dim - rot / 2) / 8), 128) == 4)
      return (int)launch_dep(retention_prepare_vec_kernel<4, 2>, dim3((T + 3) / 4), dim3(256), 4 * smem, stream,
                             (const __nv_bfloat16*)proj, ld, n_heads, dim, rot, T, k_scale, positions, inv_f, inv_d, qk, act);
    return (int)launch_dep(retention_prepare_vec_kernel<1, 1>, dim3(T), dim3(256), smem, stream, (const __nv_bfloat16*)proj, ld,
                           n_heads, dim, rot, T, k_scale, positions, inv_f, inv_d, qk, act);
  }
  if (dtype == MF_F32)
    return (int)launch_dep(retention_prepare_kernel<float>, dim3(T), dim3(256), smem, stream, (const float*)proj, ld,
                           n_heads, dim, rot, k_scale, positions, inv_f, inv_d, qk, act, v_out, v_off, nv);
  if (dtype == MF_BF16)
    return (int)launch_dep(retention_prepare_kernel<__nv_bfloat16>, dim3(T), dim3(256), smem, stream,
                           (const __nv_bfloat16*)proj, ld, n_heads, dim, rot, k_scale, positions, inv_f, inv_d, qk,
                           act, v_out, v_off, nv);
  return MF_ERR_BAD_DTYPE;
}

// qk [T, 2 heads dim] (32-bit, prepared); v read from the projections' rows (v + t * v_ld + h * vdim).
// state [slots, heads, dim, vdim] with `state_stride` floats per slot.  o_out [T, heads * vdim] 32-bit.
template <typename T, int RPL>
__global__ void __launch_bounds__(RT_THREADS)
retention_recurrence_kernel(const float* qk, const T* v, long long v_ld,
                            const float* __restrict__ decay, float* state, long long state_stride,
                            const int* seq_q_start, const int* seq_q_len,
                            const int* slots, float* __restrict__ o_out, int n_heads, int dim, int vdim) {
  extern __shared__ float sm[];            // [RT_CHUNK][2 dim] q then k of a token, [RT_CHUNK][RT_COLS] v
  float* v_s = sm + RT_CHUNK * 2 * dim;
  pdl_launch();
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * RT_COLS;
  const int lane = threadIdx.x % RT_LANES, cl = threadIdx.x / RT_LANES;
  const int c = c0 + cl;
  const bool col_ok = c < vdim;
  const int t0 = seq_q_start[s], n = seq_q_len[s];
  const float g = decay[h];
  float* S = state + (long long)slots[s] * state_stride + (long long)h * dim * vdim;
  float st[RPL];
#pragma unroll
  for (int i = 0; i < RPL; i++) {
    const int r = lane + i * RT_LANES;
    st[i] = (col_ok && r < dim) ? S[(long long)r * vdim + c] : 0.f;
  }
  for (int b = 0; b < n; b += RT_CHUNK) {
    const int nb = min(RT_CHUNK, n - b);
    __syncthreads();
    for (int i = threadIdx.x; i < nb * 2 * dim; i += RT_THREADS) {
      const int tt = i / (2 * dim), d = i - tt * 2 * dim;
      const int hh = d / dim, ch = d - hh * dim;         // 0: q, 1: k
      sm[i] = qk[(long long)(t0 + b + tt) * 2 * n_heads * dim + (long long)(hh * n_heads + h) * dim + ch];
    }
    for (int i = threadIdx.x; i < nb * RT_COLS; i += RT_THREADS) {
      const int tt = i / RT_COLS, cc = i - tt * RT_COLS;
      v_s[i] = (c0 + cc < vdim) ? to_f32<T>(v[(long long)(t0 + b + tt) * v_ld + (long long)h * vdim + c0 + cc]) : 0.f;
    }
    __syncthreads();
    for (int tt = 0; tt < nb; tt++) {
      const float* qs = sm + tt * 2 * dim;
      const float* ks = qs + dim;
      const float vc = v_s[tt * RT_COLS + cl];
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < RPL; i++) {
        const int r = lane + i * RT_LANES;
        if (r < dim) {
          st[i] = fmaf(g, st[i], ks[r] * vc);
          acc = fmaf(st[i], qs[r], acc);
        }
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      if (lane == 0 && col_ok) o_out[(long long)(t0 + b + tt) * n_heads * vdim + (long long)h * vdim + c] = acc;
    }
  }
#pragma unroll
  for (int i = 0; i < RPL; i++) {
    const int r = lane + i * RT_LANES;
    if (col_ok && r < dim) S[(long long)r * vdim + c] = st[i];
  }
}

// ---------------------------------------------------------------------------- the same, staged
// For sizes in whole pieces (dim a multiple of the rows per block, vdim of 16, 16-byte aligned rows): a block owns
// RS_ROWS rows x RT_COLS columns of S, so that a head's state is spread over dim/RS_ROWS x vdim/RT_COLS
// blocks (an element of S depends on no other element; only the read-out sums over rows, and that sum
// is finished by the output kernel over the row groups' partial read-outs).  The block's share of q, k
// and v of the coming tokens arrives through a ring of cp.async stages, RS_CHUNK tokens each, so that no
// token waits for memory.
namespace {
constexpr int RS_CHUNK = 16;
constexpr int RS_STAGES = 4;

__device__ __forceinline__ void rs_cp_async_16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
}  // namespace

template <typename T, int RS_ROWS>
__global__ void __launch_bounds__(RT_THREADS)
retention_recurrence_staged_kernel(const float* qk, const T* v, long long v_ld,
                                   const float* __restrict__ decay, float* state, long long state_stride,
                                   const int* seq_q_start, const int* seq_q_len,
                                   const int* slots, float* __restrict__ o_part, long long part_stride,
                                   int n_heads, int dim, int vdim) {
  constexpr int RS_RPL = RS_ROWS / RT_LANES;
  constexpr int V_PIECES = RT_COLS * sizeof(T) / 16;               // 16-byte pieces of a token's values
  constexpr int PIECES = 2 * RS_ROWS / 4 + V_PIECES;               // q, k, v of one token
  constexpr int TOKEN_FLOATS = 2 * RS_ROWS + RT_COLS * sizeof(T) / 4;
  __shared__ __align__(16) float ring[RS_STAGES][RS_CHUNK][TOKEN_FLOATS];
  pdl_launch();
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y;
  const int n_cb = vdim / RT_COLS;
  const int rg = blockIdx.z / n_cb, c0 = (blockIdx.z - rg * n_cb) * RT_COLS, r0 = rg * RS_ROWS;
  const int lane = threadIdx.x % RT_LANES, cl = threadIdx.x / RT_LANES;
  const int t0 = seq_q_start[s], n = seq_q_len[s];
  const float g = decay[h];
  float* S = state + (long long)slots[s] * state_stride + ((long long)h * dim + r0) * vdim + c0 + cl;
  float st[RS_RPL];
#pragma unroll
  for (int i = 0; i < RS_RPL; i++) st[i] = S[(long long)(lane + i * RT_LANES) * vdim];
  const int n_chunks = (n + RS_CHUNK - 1) / RS_CHUNK;

  auto fetch = [&](int chunk) {
    const int stage = chunk % RS_STAGES;
    const int nb = min(RS_CHUNK, n - chunk * RS_CHUNK);
    for (int i = threadIdx.x; i < nb * PIECES; i += RT_THREADS) {
      const int tt = i / PIECES, p = i - tt * PIECES;
      const long long t = t0 + chunk * RS_CHUNK + tt;
      float* dst = &ring[stage][tt][0] + p * 4;
      if (p < 2 * RS_ROWS / 4) {
        const int which = p / (RS_ROWS / 4), q4 = p - which * (RS_ROWS / 4);      // 0: q, 1: k
        rs_cp_async_16(dst, qk + t * 2 * n_heads * dim + (long long)(which * n_heads + h) * dim + r0 + q4 * 4);
      } else {
        const int v4 = p - 2 * RS_ROWS / 4;
        rs_cp_async_16(dst, reinterpret_cast<const char*>(v + t * v_ld + (long long)h * vdim + c0) + v4 * 16);
      }
    }
  };
#pragma unroll
  for (int c = 0; c < RS_STAGES - 1; c++) {
    if (c < n_chunks) fetch(c);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float* o = o_part + (long long)rg * part_stride + (long long)h * vdim + c0 + cl;
  for (int chunk = 0; chunk < n_chunks; chunk++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(RS_STAGES - 2) : "memory");
    __syncthreads();          // the chunk has landed for everyone, and everyone is done with the stage refilled next
    if (chunk + RS_STAGES - 1 < n_chunks) fetch(chunk + RS_STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const int stage = chunk % RS_STAGES;
    const int nb = min(RS_CHUNK, n - chunk * RS_CHUNK);
    // four tokens at a time: only the state is a chain from token to token; the four read-outs' sums
    // over the lanes of a column go through their shuffles side by side
    for (int tt = 0; tt < nb; tt += 4) {
      float acc[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        acc[u] = 0.f;
        if (tt + u < nb) {
          const float* qs = &ring[stage][tt + u][0];
          const float* ks = qs + RS_ROWS;
          const float vc = to_f32<T>(reinterpret_cast<const T*>(ks + RS_ROWS)[cl]);
#pragma unroll
          for (int i = 0; i < RS_RPL; i++) {
            const int r = lane + i * RT_LANES;
            st[i] = fmaf(g, st[i], ks[r] * vc);
            acc[u] = fmaf(st[i], qs[r], acc[u]);
          }
        }
      }
#pragma unroll
      for (int m = 1; m < RT_LANES; m <<= 1)
#pragma unroll
        for (int u = 0; u < 4; u++) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], m);
      if (lane == 0) {
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (tt + u < nb) o[(long long)(t0 + chunk * RS_CHUNK + tt + u) * n_heads * vdim] = acc[u];
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < RS_RPL; i++) S[(long long)(lane + i * RT_LANES) * vdim] = st[i];
}

// One token of every sequence: a block of four warps per (sequence, head, 32 columns), a column a lane, a quarter of the rows a
// warp, all of them fetched at once in whole lines of 128 bytes before the arithmetic begins; the whole read-out in one block, so
// no partial ones go through memory.  The kernels above set up a ring for one token and take half lines of the state:
// the layer's step of 8 sequences of 16 heads of 128 x 128 39.8 -> 27.4 us, of 32 sequences 68.9 -> 42.1 (17 and 67 MB there
// and back).
template <typename T, int DIM>
__global__ void __launch_bounds__(128)
retention_step_kernel(const float* qk, const T* v, long long v_ld, const float* __restrict__ decay,
                      float* state, long long state_stride, const int* seq_q_start,
                      const int* slots, float* __restrict__ o_out, int n_heads, int vdim) {
  constexpr int ROWS = DIM / 4;
  __shared__ float q_s[DIM], k_s[DIM], part[4][32];
  pdl_launch();
  pdl_wait();
  const int seq = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.z * 32 + lane;
  const long long t = seq_q_start[seq];
  float* S = state + (long long)slots[seq] * state_stride + ((long long)h * DIM + warp * ROWS) * vdim + col;
  float s[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; i++) s[i] = S[(long long)i * vdim];
  const float* row = qk + (t * 2 * n_heads + h) * DIM;
  for (int i = threadIdx.x; i < DIM; i += 128) {
    q_s[i] = row[i];
    k_s[i] = row[n_heads * DIM + i];
  }
  const float vc = to_f32<T>(v[t * v_ld + (long long)h * vdim + col]), g = decay[h];
  __syncthreads();
  const float *q = q_s + warp * ROWS, *k = k_s + warp * ROWS;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < ROWS; i++) {
    s[i] = fmaf(g, s[i], k[i] * vc);
    S[(long long)i * vdim] = s[i];
    acc[i & 3] = fmaf(s[i], q[i], acc[i & 3]);
  }
  part[warp][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  __syncthreads();
  if (warp == 0)
    o_out[(t * n_heads + h) * vdim + col] = (part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]);
}

// Rows of S per block of the staged kernel: 16, 32 or 64.  Fewer rows spread a head over more blocks,
// more rows give a thread more of S to work on per operand it fetches.
static int g_retention_rows = 32;
MF_API int mf_set_retention_rows(int rows) {
  if (rows != 16 && rows != 32 && rows != 64) return MF_ERR_BAD_ARG;
  g_retention_rows = rows;
  return 0;
}

// How many partial read-outs (row groups) a launch writes: retention_output sums them.
MF_API int mf_retention_parts(int dim, int vdim, int v_dtype, long long v_ld) {
  const int vb = v_dtype == MF_F32 ? 4 : 2;
  const bool staged = dim % g_retention_rows == 0 && vdim % RT_COLS == 0 && (v_ld * vb) % 16 == 0 &&
                      (vdim * vb) % 16 == 0;
  return staged ? dim / g_retention_rows : 1;
}

template <typename T, int ROWS>
static int launch_staged(const float* qk, const void* v, long long v_ld, const float* decay, float* state,
                         long long state_stride, const int* seq_q_start, const int* seq_q_len, const int* slots,
                         float* o_out, long long part_stride, int n_seqs, int n_heads, int dim, int vdim,
                         cudaStream_t stream) {
  dim3 grid(n_seqs, n_heads, (dim / ROWS) * (vdim / RT_COLS));
  return (int)launch_dep(retention_recurrence_staged_kernel<T, ROWS>, grid, dim3(RT_THREADS), 0, stream, qk, (const T*)v,
                         v_ld, decay, state, state_stride, seq_q_start, seq_q_len, slots, o_out, part_stride, n_heads,
                         dim, vdim);
}

// Whether a step of one token a sequence has a kernel of its own for these sizes (one read-out, no partial ones).
MF_API int mf_retention_step_ok(int dim, int vdim) { return (dim == 64 || dim == 128) && vdim > 0 && vdim % 32 == 0; }

// `one_each`: every sequence brings exactly one token, mf_retention_step_ok says yes, and o_out holds one read-out.
MF_API int mf_retention_recurrence(const float* qk, const void* v, int v_dtype, long long v_ld, const float* decay,
                                   float* state, long long state_stride, const int* seq_q_start,
                                   const int* seq_q_len, const int* slots, float* o_out, long long part_stride,
                                   int n_seqs, int one_each, int n_heads, int dim, int vdim, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (dim <= 0 || dim > 64 * RT_LANES || vdim <= 0 || n_heads <= 0 || n_heads > 65535) return MF_ERR_BAD_ARG;
  if (one_each) {
    if (!mf_retention_step_ok(dim, vdim)) return MF_ERR_BAD_ARG;
    if (v_dtype != MF_F32 && v_dtype != MF_BF16) return MF_ERR_BAD_DTYPE;
    mf_count(MF_K_RETENTION_RECURRENCE);
    mf_count(MF_K_RETENTION_STEP);
    const dim3 step_grid(n_seqs, n_heads, vdim / 32);
    if (v_dtype == MF_F32)
      return (int)launch_dep(dim == 64 ? retention_step_kernel<float, 64> : retention_step_kernel<float, 128>, step_grid,
                             dim3(128), 0, stream, qk, (const float*)v, v_ld, decay, state, state_stride, seq_q_start, slots,
                             o_out, n_heads, vdim);
    return (int)launch_dep(dim == 64 ? retention_step_kernel<__nv_bfloat16, 64> : retention_step_kernel<__nv_bfloat16, 128>,
                           step_grid, dim3(128), 0, stream, qk, (const __nv_bfloat16*)v, v_ld, decay, state, state_stride,
                           seq_q_start, slots, o_out, n_heads, vdim);
  }
  // o_out holds mf_retention_parts(...) partial read-outs, `part_stride` floats apart
  if (mf_retention_parts(dim, vdim, v_dtype, v_ld) > 1 && ((uintptr_t)qk & 15) == 0 && ((uintptr_t)v & 15) == 0 &&
      (v_dtype == MF_F32 || v_dtype == MF_BF16)) {
    mf_count(MF_K_RETENTION_RECURRENCE);
#define RS_GO(TT, ROWS)                                                                                             \
  return launch_staged<TT, ROWS>(qk, v, v_ld, decay, state, state_stride, seq_q_start, seq_q_len, slots, o_out,     \
                                 part_stride, n_seqs, n_heads, dim, vdim, stream)
#define RS_ROWS_PICK(TT)                  \
  if (g_retention_rows == 16) RS_GO(TT, 16); \
  if (g_retention_rows == 32) RS_GO(TT, 32); \
  RS_GO(TT, 64)
    if (v_dtype == MF_F32) { RS_ROWS_PICK(float); }
    RS_ROWS_PICK(__nv_bfloat16);
#undef RS_ROWS_PICK
#undef RS_GO
  }
  if (mf_retention_parts(dim, vdim, v_dtype, v_ld) > 1) return MF_ERR_BAD_ARG;     // the caller sized o_out for parts
  dim3 grid(n_seqs, n_heads, (vdim + RT_COLS - 1) / RT_COLS);
  const size_t smem = (size_t)RT_CHUNK * (2 * dim + RT_COLS) * sizeof(float);
  const int per = (dim + RT_LANES - 1) / RT_LANES;
  mf_count(MF_K_RETENTION_RECURRENCE);
#define RT_LAUNCH(TT, RPL)                                                                                       \
  return (int)launch_dep(retention_recurrence_kernel<TT, RPL>, grid, dim3(RT_THREADS), smem, stream, qk,         \
                         (const TT*)v, v_ld, decay, state, state_stride, seq_q_start, seq_q_len, slots, o_out,   \
                         n_heads, dim, vdim)
#define RT_PICK(TT)              \
  if (per <= 4) RT_LAUNCH(TT, 4);  \
  if (per <= 8) RT_LAUNCH(TT, 8);  \
  if (per <= 16) RT_LAUNCH(TT, 16); \
  if (per <= 32) RT_LAUNCH(TT, 32); \
  RT_LAUNCH(TT, 64)
  if (v_dtype == MF_F32) { RT_PICK(float); }
  if (v_dtype == MF_BF16) { RT_PICK(__nv_bfloat16); }
#undef RT_PICK
#undef RT_LAUNCH
  return MF_ERR_BAD_DTYPE;
}

// out[t, h, :] = o[t, h, :] / sqrt(mean(o[t, h, :]^2) + eps) * silu(gate[t, h, :]); a warp per (token, head).
// whole: one root mean square over all heads of the token instead of one per head.  weight (optional):
// [n_heads * vdim], multiplied in.  gate_act 1: the gate passes a sigmoid instead of SiLU.
template <typename T>
__global__ void retention_output_kernel(const float* o, int n_parts, long long part_stride,
                                        const T* gate, long long gate_ld, float eps, T* __restrict__ out,
                                        int n_heads, int vdim, const float* __restrict__ weight, int whole,
                                        int gate_act) {
  extern __shared__ float ro_ss[];      // [n_heads] sums of squares
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  auto read = [&](const float* orow, int d) {
    // the read-out is the sum of the row groups' partial read-outs, added in their order
    float v = orow[d];
    for (int p = 1; p < n_parts; p++) v += orow[p * part_stride + d];
    return v;
  };
  for (int h = warp; h < n_heads; h += nw) {
    const float* orow = o + ((long long)t * n_heads + h) * vdim;
    float ss = 0.f;
    for (int d = lane; d < vdim; d += 32) {
      const float v = read(orow, d);
      ss += v * v;
    }
    ss = warp_sum(ss);
    if (lane == 0) ro_ss[h] = ss;
  }
  __syncthreads();
  float all = 0.f;
  if (whole)
    for (int h = 0; h < n_heads; h++) all += ro_ss[h];
  for (int h = warp; h < n_heads; h += nw) {
    const float* orow = o + ((long long)t * n_heads + h) * vdim;
    const T* grow = gate + (long long)t * gate_ld + (long long)h * vdim;
    const float inv = whole ? 1.0f / sqrtf(all / (float)(n_heads * vdim) + eps) : 1.0f / sqrtf(ro_ss[h] / (float)vdim + eps);
    T* dst = out + ((long long)t * n_heads + h) * vdim;
    for (int d = lane; d < vdim; d += 32) {
      const float g = to_f32<T>(grow[d]);
      const float sg = 1.0f / (1.0f + expf(-g));
      const float w = weight ? weight[h * vdim + d] : 1.0f;
      dst[d] = from_f32<T>(read(orow, d) * inv * w * (gate_act ? sg : g * sg));
    }
  }
}

// The same where the norm is per head and a head is 32 N columns in whole pieces: a warp per (token, head), N neighbouring columns a
// lane, read once and kept.  1,777 tokens of 8 heads of 128: 8.9 us with a block per token that reads twice, 5.6 here.
template <typename T, int N>
__global__ void __launch_bounds__(256)
retention_output_vec_kernel(const float* o, int n_parts, long long part_stride, const T* gate,
                            long long gate_ld, float eps, T* __restrict__ out, int n_heads, int total,
                            const float* __restrict__ weight, int gate_act) {
  constexpr int V = 32 * N;
  pdl_launch();
  pdl_wait();
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), d = (threadIdx.x & 31) * N;
  if (item >= total) return;
  const int t = item / n_heads, h = item - t * n_heads;
  const float* orow = o + (long long)item * V + d;
  const T* grow = gate + (long long)t * gate_ld + (long long)h * V + d;
  struct alignas(4 * N) F { float x[N]; };
  struct alignas(sizeof(T) * N) G { T x[N]; };
  const G g = *reinterpret_cast<const G*>(grow);
  F v = *reinterpret_cast<const F*>(orow);
  for (int p = 1; p < n_parts; p++) {      // the row groups' partial read-outs, added in their order
    const F w = *reinterpret_cast<const F*>(orow + p * part_stride);
#pragma unroll
    for (int i = 0; i < N; i++) v.x[i] += w.x[i];
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < N; i++) ss += v.x[i] * v.x[i];
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)V + eps);
  G r;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float gi = to_f32<T>(g.x[i]), sg = 1.0f / (1.0f + expf(-gi));
    const float w = weight ? weight[h * V + d + i] : 1.0f;
    r.x[i] = from_f32<T>(v.x[i] * inv * w * (gate_act ? sg : gi * sg));
  }
  *reinterpret_cast<G*>(out + (long long)item * V + d) = r;
}

MF_API int mf_retention_output(const float* o, int n_parts, long long part_stride, const void* gate, int dtype,
                               long long gate_ld, float eps, void* out, int T, int n_heads, int vdim,
                               const float* weight, int whole, int gate_act, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (n_parts < 1) return MF_ERR_BAD_ARG;
  mf_count(MF_K_RETENTION_OUTPUT);
  if (!whole && n_heads > 0 && (vdim == 64 || vdim == 128) && (dtype == MF_F32 || dtype == MF_BF16) && (long long)T * n_heads < (1ll << 31) - 8 &&
      gate_ld % 4 == 0 && part_stride % 4 == 0 && !(((uintptr_t)o | (uintptr_t)gate | (uintptr_t)out) & 15)) {
    const dim3 grid((unsigned)(((long long)T * n_heads + 7) / 8));
#define RO_GO(TT, N)                                                                                                     \
  return (int)launch_dep(retention_output_vec_kernel<TT, N>, grid, dim3(256), 0, stream, o, n_parts, part_stride,        \
                         (const TT*)gate, gate_ld, eps, (TT*)out, n_heads, T * n_heads, weight, gate_act)
    if (dtype == MF_F32) {
      if (vdim == 64) RO_GO(float, 2);
      RO_GO(float, 4);
    }
    if (vdim == 64) RO_GO(__nv_bfloat16, 2);
    RO_GO(__nv_bfloat16, 4);
#undef RO_GO
  }
  const int threads = n_heads >= 8 ? 256 : 32 * (n_heads > 0 ? n_heads : 1);
  const size_t smem = (size_t)(n_heads > 0 ? n_heads : 1) * sizeof(float);
  if (smem > 48 * 1024) return MF_ERR_BAD_ARG;
  if (dtype == MF_F32)
    return (int)launch_dep(retention_output_kernel<float>, dim3(T), dim3(threads), smem, stream, o, n_parts, part_stride,
                           (const float*)gate, gate_ld, eps, (float*)out, n_heads, vdim, weight, whole, gate_act);
  if (dtype == MF_BF16)
    return (int)launch_dep(retention_output_kernel<__nv_bfloat16>, dim3(T), dim3(threads), smem, stream, o, n_parts,
                           part_stride, (const __nv_bfloat16*)gate, gate_ld, eps, (__nv_bfloat16*)out, n_heads, vdim,
                           weight, whole, gate_act);
  return MF_ERR_BAD_DTYPE;
}
