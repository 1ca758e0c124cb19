// Rotary position encoding in either pairing, fused with the write of keys and values into
// their pages, for mixers whose values are their keys as projected (before the rotation).
//
// One block per token.  A row of `qk` (rows `ld` elements apart) holds the query heads, then the key heads, then (unless the
// values are the keys) the value heads, each head_dim wide.  The first `rot` channels of every
// query and key head are rotated, pair j by the angle position * inv[j]: the pair (u, v) becomes
// (u cos a - v sin a, v cos a + u sin a); the other channels pass.  Rotated queries go to q_out
// [T, n_heads * head_dim], rotated keys to the key pages, and the value pages get the keys before
// the rotation (v_from_k) or the row's value heads.
#include "rotary.cuh"

template <typename T>
__global__ void rope_store_kernel(const T* qk, int ld, int n_heads, int n_kv, int hd, int rot, int layout,
                                  const int* positions, const int* seq_of_token,
                                  PagedView pv, const float* __restrict__ inv_f, const double* __restrict__ inv_d,
                                  T* __restrict__ q_out, T* __restrict__ k_pool, T* __restrict__ v_pool,
                                  int write_kv, int v_from_k) {
  extern __shared__ float cs[];            // [half] cos, [half] sin
  pdl_launch();
  const int t = blockIdx.x;
  const int pos = positions[t], seq = seq_of_token[t];
  const int half = rot >> 1;
  for (int j = threadIdx.x; j < half; j += blockDim.x) rotary_cs(pos, j, inv_f, inv_d, cs[j], cs[half + j]);
  __syncthreads();
  pdl_wait();
  const T* row = qk + (long long)t * ld;
  const int per_head = hd - half;          // `half` pairs and hd - rot channels that pass
  const int heads = n_heads + (write_kv ? n_kv : 0);
  for (int idx = threadIdx.x; idx < heads * per_head; idx += blockDim.x) {
    const int h = idx / per_head, j = idx - h * per_head;
    const T* src = row + (long long)h * hd;
    const bool is_k = h >= n_heads;
    const long long off = is_k ? paged_offset(pv, seq, pos, h - n_heads) : 0;
    T* dst = is_k ? k_pool + off : q_out + ((long long)t * n_heads + h) * hd;
    T* vdst = (is_k && v_from_k) ? v_pool + off : nullptr;
    if (j < half) {
      int a, b;
      rotary_pair(layout, rot, j, a, b);
      const float c = cs[j], s = cs[half + j];
      const float u = to_f32<T>(src[a]), v = to_f32<T>(src[b]);
      dst[a] = from_f32<T>(u * c - v * s);
      dst[b] = from_f32<T>(v * c + u * s);
      if (vdst) {
        vdst[a] = src[a];
        vdst[b] = src[b];
      }
    } else {
      const int ch = rot + (j - half);
      dst[ch] = src[ch];
      if (vdst) vdst[ch] = src[ch];
    }
  }
  if (write_kv && !v_from_k) {
    for (int idx = threadIdx.x; idx < n_kv * hd; idx += blockDim.x) {
      const int h = idx / hd, ch = idx - h * hd;
      v_pool[paged_offset(pv, seq, pos, h) + ch] = row[(long long)(n_heads + n_kv + h) * hd + ch];
    }
  }
}

// bfloat16 with adjacent pairs (2i, 2i + 1), an even head size: a pair is one 32-bit word, and so
// are two channels that pass; every thread moves whole words.
__global__ void __launch_bounds__(256)
rope_store_pairs_bf16_kernel(const __nv_bfloat16* qk, int ld, int n_heads, int n_kv, int hd, int rot,
                             const int* positions, const int* seq_of_token, PagedView pv,
                             const float* __restrict__ inv_f, __nv_bfloat16* __restrict__ q_out,
                             __nv_bfloat16* __restrict__ k_pool, __nv_bfloat16* __restrict__ v_pool, int write_kv) {
  extern __shared__ float cs[];            // [half] cos, [half] sin
  pdl_launch();
  const int t = blockIdx.x;
  const int pos = positions[t], seq = seq_of_token[t];
  const int half = rot >> 1, words = hd >> 1;
  for (int j = threadIdx.x; j < half; j += blockDim.x) sincosf((float)pos * inv_f[j], &cs[half + j], &cs[j]);
  __syncthreads();
  pdl_wait();
  const __nv_bfloat16* row = qk + (long long)t * ld;
  const int heads = n_heads + (write_kv ? n_kv : 0);
  for (int idx = threadIdx.x; idx < heads * words; idx += blockDim.x) {
    const int h = idx / words, j = idx - h * words;
    const __nv_bfloat162 in = *reinterpret_cast<const __nv_bfloat162*>(row + (long long)h * hd + 2 * j);
    __nv_bfloat162 o = in;
    if (j < half) {
      const float2 f = __bfloat1622float2(in);
      const float c = cs[j], s = cs[half + j];
      o = __floats2bfloat162_rn(f.x * c - f.y * s, f.y * c + f.x * s);
    }
    if (h < n_heads) {
      *reinterpret_cast<__nv_bfloat162*>(q_out + ((long long)t * n_heads + h) * hd + 2 * j) = o;
    } else {
      const long long off = paged_offset(pv, seq, pos, h - n_heads) + 2 * j;
      *reinterpret_cast<__nv_bfloat162*>(k_pool + off) = o;
      *reinterpret_cast<__nv_bfloat162*>(v_pool + off) = in;          // the values are the keys as projected
    }
  }
}

// The same in pieces of 16 bytes (head size and rotated channels multiples of 8, 16-byte aligned rows), TOK tokens a block
// (mf_store_tokens), the angles of all of them side by side.  2,048 tokens of 16 + 4 heads of 128 (23 MB, in L2): 9.5 us with a word a thread,
// 5.2 here.  One token a block has nothing to gain from several pieces a thread at once (5.2 with one, 6.5 with four).
template <int TOK, int U>
__global__ void __launch_bounds__(256)
rope_store_pairs_vec_kernel(const __nv_bfloat16* qk, int ld, int n_heads, int n_kv, int hd, int rot, int T,
                            const int* positions, const int* seq_of_token, PagedView pv,
                            const float* __restrict__ inv_f, __nv_bfloat16* __restrict__ q_out,
                            __nv_bfloat16* __restrict__ k_pool, __nv_bfloat16* __restrict__ v_pool, int write_kv) {
  extern __shared__ float cs[];            // [TOK][half] cos, then sin
  __shared__ int pos_s[TOK], seq_s[TOK];
  pdl_launch();
  const int t0 = blockIdx.x * TOK, nt = TOK == 1 ? 1 : min(TOK, T - t0), half = rot >> 1;
  if (threadIdx.x < nt) {
    pos_s[threadIdx.x] = positions[t0 + threadIdx.x];
    seq_s[threadIdx.x] = seq_of_token[t0 + threadIdx.x];
  }
  for (int i = threadIdx.x; i < nt * half; i += 256) {
    const int t = TOK == 1 ? 0 : i / half, j = i - t * half;
    sincosf((float)positions[t0 + t] * inv_f[j], &cs[TOK * half + i], &cs[i]);
  }
  __syncthreads();
  pdl_wait();
  const int pieces = hd >> 3, per_token = (n_heads + (write_kv ? n_kv : 0)) * pieces;
  // U pieces a thread are on their way before the first is stored
  for (int i0 = threadIdx.x; i0 < nt * per_token; i0 += U * 256) {
    uint4 in[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * 256, t = TOK == 1 ? 0 : i / per_token;
      if (i < nt * per_token) in[u] = *reinterpret_cast<const uint4*>(qk + (long long)(t0 + t) * ld + (i - t * per_token) * 8);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * 256, t = TOK == 1 ? 0 : i / per_token, rest = i - t * per_token;
      const int h = rest / pieces, ch = (rest - h * pieces) * 8;
      if (i >= nt * per_token) continue;
      uint4 o = in[u];
      if (ch < rot) {
        const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&in[u]);
        __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float2 f = __bfloat1622float2(a[e]);
          const float c = cs[t * half + ch / 2 + e], s = cs[(TOK + t) * half + ch / 2 + e];
          b[e] = __floats2bfloat162_rn(f.x * c - f.y * s, f.y * c + f.x * s);
        }
      }
      if (h < n_heads) {
        *reinterpret_cast<uint4*>(q_out + ((long long)(t0 + t) * n_heads + h) * hd + ch) = o;
      } else {
        const long long off = paged_offset(pv, seq_s[t], pos_s[t], h - n_heads) + ch;
        *reinterpret_cast<uint4*>(k_pool + off) = o;
        *reinterpret_cast<uint4*>(v_pool + off) = in[u];       // the values are the keys as projected
      }
    }
  }
}

MF_API int mf_rope_store(const void* qk, int ld, int dtype, int T, int n_heads, int n_kv, int hd, int rot, int layout,
                         const int* positions, const int* seq_of_token, const int* block_table, int bt_stride,
                         int page_size, const float* inv_f, const double* inv_d, void* q_out, void* k_pool,
                         void* v_pool, int write_kv, int v_from_k, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (rot < 0 || rot > hd || (rot & 1) || (layout != MF_ROT_HALF && layout != MF_ROT_PAIRS)) return MF_ERR_BAD_ARG;
  if (rot > 0 && !inv_f && !inv_d) return MF_ERR_BAD_ARG;
  PagedView pv{block_table, bt_stride, page_size, n_kv, hd};
  const size_t smem = (size_t)(rot > 0 ? rot : 1) * sizeof(float);
  mf_count(MF_K_ROPE_STORE);
  if (dtype == MF_BF16 && layout == MF_ROT_PAIRS && v_from_k && !inv_d && hd % 8 == 0 && rot % 8 == 0 && ld % 8 == 0 &&
      4 * smem <= 48 * 1024 && (((uintptr_t)qk | (uintptr_t)q_out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0) {
#define PAIRS_GO(TOK, U)                                                                                                 \
  return (int)launch_dep(rope_store_pairs_vec_kernel<TOK, U>, dim3((T + TOK - 1) / TOK), dim3(256), TOK * smem, stream,  \
                         (const __nv_bfloat16*)qk, ld, n_heads, n_kv, hd, rot, T, positions, seq_of_token, pv, inv_f, \
                         (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, write_kv)
    if (mf_store_tokens(T, (n_heads + (write_kv ? n_kv : 0)) * hd / 8) == 4) PAIRS_GO(4, 4);
    PAIRS_GO(1, 1);
#undef PAIRS_GO
  }
  if (dtype == MF_BF16 && layout == MF_ROT_PAIRS && v_from_k && !inv_d && hd % 2 == 0 && ld % 2 == 0 &&
      (((uintptr_t)qk | (uintptr_t)q_out | (uintptr_t)k_pool | (uintptr_t)v_pool) & 3) == 0)
    return (int)launch_dep(rope_store_pairs_bf16_kernel, dim3(T), dim3(256), smem, stream, (const __nv_bfloat16*)qk, ld,
                           n_heads, n_kv, hd, rot, positions, seq_of_token, pv, inv_f, (__nv_bfloat16*)q_out,
                           (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, write_kv);
  if (dtype == MF_F32)
    return (int)launch_dep(rope_store_kernel<float>, dim3(T), dim3(256), smem, stream, (const float*)qk, ld, n_heads, n_kv,
                           hd, rot, layout, positions, seq_of_token, pv, inv_f, inv_d, (float*)q_out, (float*)k_pool,
                           (float*)v_pool, write_kv, v_from_k);
  if (dtype == MF_BF16)
    return (int)launch_dep(rope_store_kernel<__nv_bfloat16>, dim3(T), dim3(256), smem, stream,
                           (const __nv_bfloat16*)qk, ld, n_heads, n_kv, hd, rot, layout, positions, seq_of_token, pv, inv_f,
                           inv_d, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, write_kv,
                           v_from_k);
  return MF_ERR_BAD_DTYPE;
}
