// Talking heads over portions of prompts: what attention_talking_tc.cu needs of attention_talking_prompt.cu.
#pragma once
#include "common.cuh"

// keys that the newest query of a sequence of `ctx` tokens sees at most
__host__ __device__ inline int talking_prompt_keys(int ctx, int window, int chunk) {
  if (window > 0 && window < ctx) ctx = window;
  return chunk > 0 && chunk < ctx ? chunk : ctx;
}
// From how many of them the kernel is the faster one (layer's attention, us, one portion, this kernel / the one of attention_talking_tc.cu):
// 16 heads, 128 keys 26.8 / 28.8 where they fill its one tile of keys, 150 keys 37.0 / 33.6, 200 keys 37.0 / 39.1, 300 keys 47 / 56, 2,048 keys
// 111 / 215; 8 heads, 64 keys 16.1 / 15.6, 100 keys 16.5 / 19.9, 300 keys 25 / 45.
inline int talking_prompt_from(int n_heads) { return n_heads == 16 ? 192 : 80; }

// Whether it takes these sizes (what else mf_attention_talking_tc takes has been checked).
bool talking_prompt_takes(int n_heads, int n_kv, int dim, int vdim, const void* q, const void* k_pool, const void* v_pool,
                          long long pool_rows);
// Cuts of a launch for which the caller has scratch for `splits` (0: none): as few as the lane's mask allows.
int talking_prompt_cuts(int splits, int chunk);
// Sequences whose queries see fewer than `from_keys` keys are left out.
int talking_prompt_launch(const void* q, const void* k_pool, const void* v_pool, void* out, const int* seq_q_start, const int* seq_q_len,
                          const int* seq_ctx_len, int table_row0, int n_seqs, int max_q_len, int n_heads, const int* block_table, int bt_stride,
                          int page_size, long long pool_rows, float scale, float softcap, const float* talk, int window, int chunk, int cuts,
                          int from_keys, float* part_o, float* part_ml, int* status, cudaStream_t stream);
