// Experts for many tokens: the (token, choice) pairs are ordered by expert and every expert's
// pairs go through tensor-core tiles, so an expert's matrices are read once per tile of 64 pairs
// instead of once per pair.  The formulas are those of moe.cu.
//
//   mf_moe_sort     one block: counts per expert, offsets, a row for every pair (slot_of), the
//                   token of every row (row_token), and the list of tiles (expert, first row, rows).
//                   Pairs whose expert is `n_real` or above (identity experts, which have no
//                   matrices) get no row: slot_of is -1 for them.
//                   Which row a pair gets inside its expert's range is not fixed, and need not be:
//                   every row is computed by itself, and the sum over a token's experts is taken in
//                   the order of the choice by the combine kernel.
//   moe_gather_launch  the tokens' rows copied into the order of the rows, for the products of moe_grouped_tc.cu, which
//                   are the ones that run unless the tiles here are asked for.
//   mf_moe_grouped_up    act[row] = g sigmoid(alpha g) (u + 1) with g, u the clamped gate and up
//                   products of the row's token (gathered by row_token), bfloat16.
//   mf_moe_grouped_down  y[row] = Wd_e act[row], 32-bit.
//
// Both products are mma.sync m16n8k16 tiles of 64 rows x 64 columns, four warps, K in steps of 64
// through two cp.async stages of shared memory: the next step's operands are on their way while
// this step's are multiplied.  The launches cover the largest possible number of tiles (known on the
// host: pairs / 64 + experts); blocks beyond the count the sort kernel wrote return at once, so a
// step's launches do not depend on its data.
#include "common.cuh"

#define MG_BM 64
#define MG_BN 64
#define MG_BK 64
#define MG_LD (MG_BK + 8)
#define MG_STAGES 2
#define MG_MAX_EXPERTS 1024
#define MG_SORT_STAGED 32768       // pairs whose tokens the sort keeps in shared memory

__device__ __forceinline__ void mg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// meta: [0] number of tiles; tiles: [max_tiles][3] = expert, first row, rows.  An expert's rows are cut into as few tiles of at
// most `tile_rows` as hold them: full ones and a rest (64 rows), or for larger tiles equal ones in steps of 16.  A thread per
// expert: offsets by a scan over the block (a thread that walked the experts alone took most of 21 us for 64 of them).
// The pairs are counted, then placed, the counts' old values asked for by nobody (a count that hands out the places at once has no second pass, but 8,192
// pairs of 16 experts wait for one another: 6.2 us, 4.7 here).  The rows' tokens are put in order in shared memory where they fit: a warp's 32
// scattered words are 32 stores to memory (12,288 pairs of 64 experts 9.6 -> 6.6 us, 384 the same 2.6).
template <bool STAGED>
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int* ids, int n_pairs, int E, int top, int tile_rows, int* slot_of,
                int* __restrict__ row_token, int* __restrict__ meta, int* __restrict__ tiles) {
  extern __shared__ int tokens[];            // STAGED: [n_pairs], a row's token
  __shared__ int count[MG_MAX_EXPERTS], cursor[MG_MAX_EXPERTS];
  __shared__ int2 warp_total[32];
  __shared__ int used_rows;
  const int e = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  pdl_launch();
  pdl_wait();
  count[e] = 0;
  __syncthreads();
  // eight pairs a thread at a time: their loads are on their way together; the first eight stay in registers
  constexpr int AT_ONCE = 8;
  int held[AT_ONCE];
#pragma unroll
  for (int k = 0; k < AT_ONCE; k++) held[k] = e + k * 1024 < n_pairs ? ids[e + k * 1024] : -1;
#pragma unroll
  for (int k = 0; k < AT_ONCE; k++)
    if (held[k] >= 0 && held[k] < E) atomicAdd(&count[held[k]], 1);
  for (int i0 = e + AT_ONCE * 1024; i0 < n_pairs; i0 += AT_ONCE * 1024) {
    int own[AT_ONCE];
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) own[k] = i0 + k * 1024 < n_pairs ? ids[i0 + k * 1024] : E;
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++)
      if (own[k] < E) atomicAdd(&count[own[k]], 1);
  }
  __syncthreads();
  {
    const int n = count[e], nt = (n + tile_rows - 1) / tile_rows;
    int rows = n, blocks = nt;               // inclusive sums over the experts up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, rows, o), b = __shfl_up_sync(0xffffffffu, blocks, o);
      if (lane >= o) {
        rows += a;
        blocks += b;
      }
    }
    if (lane == 31) warp_total[warp] = make_int2(rows, blocks);
    __syncthreads();
    int2 before = make_int2(0, 0);
    for (int w = 0; w < warp && w * 32 < E; w++) {      // warps beyond the experts hold none
      before.x += warp_total[w].x;
      before.y += warp_total[w].y;
    }
    rows += before.x;
    blocks += before.y;
    cursor[e] = rows - n;                    // the expert's first row
    if (e == E - 1) {
      meta[0] = blocks;
      used_rows = rows;
    }
    const int per = tile_rows <= MG_BM ? tile_rows : (nt > 0 ? ((n + nt - 1) / nt + 15) / 16 * 16 : 0);
    for (int k = 0; k < nt; k++) {
      int* t = tiles + 3 * (blocks - nt + k);
      t[0] = e;
      t[1] = rows - n + k * per;
      t[2] = max(0, min(per, n - k * per));
    }
  }
  __syncthreads();
  auto put = [&](int i, int id) {
    if (id < 0) return;
    if (id >= E) {              // an identity expert: no row
      slot_of[i] = -1;
      return;
    }
    const int row = atomicAdd(&cursor[id], 1);
    slot_of[i] = row;
    if (STAGED) tokens[row] = i / top;
    else row_token[row] = i / top;
  };
#pragma unroll
  for (int k = 0; k < AT_ONCE; k++) put(e + k * 1024, held[k]);
  for (int i0 = e + AT_ONCE * 1024; i0 < n_pairs; i0 += AT_ONCE * 1024) {
    int own[AT_ONCE];
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) own[k] = i0 + k * 1024 < n_pairs ? ids[i0 + k * 1024] : -1;
#pragma unroll
    for (int k = 0; k < AT_ONCE; k++) put(i0 + k * 1024, own[k]);
  }
  if (STAGED) {
    __syncthreads();
    for (int i = threadIdx.x; i < used_rows; i += blockDim.x) row_token[i] = tokens[i];
  }
  // rows that no pair took (pairs of identity experts have none) name token 0, so that a gather over all
  // n_pairs rows stays inside x
  for (int i = used_rows + threadIdx.x; i < n_pairs; i += blockDim.x) row_token[i] = 0;
}

MF_API int mf_moe_sort(const int* ids, int T, int E, int top, int tile_rows, int* slot_of, int* row_token, int* meta,
                       int* tiles, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (E < 1 || E > MG_MAX_EXPERTS || tile_rows < MG_BM || tile_rows % 16) return MF_ERR_BAD_ARG;
  mf_count(MF_K_MOE_SORT);
  const int n = T * top;
  if (n > MG_SORT_STAGED)
    return (int)launch_dep(moe_sort_kernel<false>, dim3(1), dim3(1024), 0, stream, ids, n, E, top, tile_rows, slot_of, row_token,
                           meta, tiles);
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    const cudaError_t e =
        cudaFuncSetAttribute(moe_sort_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SORT_STAGED * 4);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  return (int)launch_dep(moe_sort_kernel<true>, dim3(1), dim3(1024), n * sizeof(int), stream, ids, n, E, top, tile_rows, slot_of,
                         row_token, meta, tiles);
}

__device__ __forceinline__ void mg_ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mg_cp16(void* smem, const void* gmem) {
  const uint32_t addr = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(addr), "l"(gmem) : "memory");
}

// One 64 x 64 tile: acc += A[64 rows, K] * B[64 rows of W, K]^T, A rows given by pointers.
// `arow(r)` -> pointer to row r of A (or null), `brow(n)` -> pointer to row n of W (or null).
// As: [MG_STAGES][64][MG_LD], Bs: [MG_STAGES][NB * 64][MG_LD].
template <int NB, typename ARow, typename BRow>
__device__ __forceinline__ void mg_tile(float (&acc)[NB][MG_BN / 8][4], int K, ARow arow, BRow brow,
                                        __nv_bfloat16* As, __nv_bfloat16* Bs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto load = [&](int k0, int stage) {
    __nv_bfloat16* Ad = As + (size_t)stage * MG_BM * MG_LD;
    __nv_bfloat16* Bd = Bs + (size_t)stage * NB * MG_BN * MG_LD;
    for (int i = tid; i < MG_BM * (MG_BK / 8); i += blockDim.x) {
      const int r = i / (MG_BK / 8), c = (i - r * (MG_BK / 8)) * 8;
      const __nv_bfloat16* p = arow(r);
      if (p && k0 + c < K) mg_cp16(Ad + r * MG_LD + c, p + k0 + c);
      else *reinterpret_cast<uint4*>(Ad + r * MG_LD + c) = make_uint4(0, 0, 0, 0);
    }
    for (int i = tid; i < NB * MG_BN * (MG_BK / 8); i += blockDim.x) {
      const int n = i / (MG_BK / 8), c = (i - n * (MG_BK / 8)) * 8;
      const __nv_bfloat16* p = brow(n);
      if (p && k0 + c < K) mg_cp16(Bd + n * MG_LD + c, p + k0 + c);
      else *reinterpret_cast<uint4*>(Bd + n * MG_LD + c) = make_uint4(0, 0, 0, 0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  load(0, 0);
  int stage = 0;
  for (int k0 = 0; k0 < K; k0 += MG_BK, stage ^= 1) {
    if (k0 + MG_BK < K) {
      load(k0 + MG_BK, stage ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const __nv_bfloat16* Ac = As + (size_t)stage * MG_BM * MG_LD;
    const __nv_bfloat16* Bc = Bs + (size_t)stage * NB * MG_BN * MG_LD;
#pragma unroll
    for (int kk = 0; kk < MG_BK; kk += 16) {
      // fragments by ldmatrix: A's four 8x8 blocks in one load, B's blocks of two column tiles in one
      uint32_t af[4];
      mg_ldmatrix_x4(af, Ac + (warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * MG_LD + kk + (lane >> 4) * 8);
#pragma unroll
      for (int b = 0; b < NB; b++) {
#pragma unroll
        for (int nt = 0; nt < MG_BN / 8; nt += 2) {
          uint32_t bf[4];
          mg_ldmatrix_x4(bf, Bc + (b * MG_BN + nt * 8 + (lane & 7) + (lane >> 4) * 8) * MG_LD + kk + ((lane >> 3) & 1) * 8);
          mg_mma(acc[b][nt], af, bf[0], bf[1]);
          mg_mma(acc[b][nt + 1], af, bf[2], bf[3]);
        }
      }
    }
    __syncthreads();       // the stage is read: the load after the next may overwrite it
  }
}

// NB 2: gate and up tiles side by side and the gated activation; NB 1: an expert without a gate, whose
// first matrix is [ff, H] alone, and the activation `act_kind` of its sums.
template <int NB>
__global__ void __launch_bounds__(128)
moe_grouped_up_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w_gu,
                      const int* __restrict__ row_token, const int* __restrict__ meta, const int* __restrict__ tiles,
                      __nv_bfloat16* __restrict__ act, int H, int ff, float limit, float alpha, float up_off,
                      int act_kind) {
  extern __shared__ __align__(16) __nv_bfloat16 mg_smem[];
  __nv_bfloat16* As = mg_smem;
  __nv_bfloat16* Bs = mg_smem + MG_STAGES * MG_BM * MG_LD;
  if ((int)blockIdx.x >= meta[0]) return;
  const int e = tiles[3 * blockIdx.x], row_first = tiles[3 * blockIdx.x + 1], rows = tiles[3 * blockIdx.x + 2];
  const int n0 = blockIdx.y * MG_BN;
  const __nv_bfloat16* wg = w_gu + (long long)e * NB * ff * H;
  const __nv_bfloat16* wu = wg + (long long)ff * H;
  float acc[NB][MG_BN / 8][4];
#pragma unroll
  for (int b = 0; b < NB; b++)
#pragma unroll
    for (int nt = 0; nt < MG_BN / 8; nt++) acc[b][nt][0] = acc[b][nt][1] = acc[b][nt][2] = acc[b][nt][3] = 0.f;
  mg_tile<NB>(acc, H,
             [&](int r) { return r < rows ? x + (long long)row_token[row_first + r] * H : nullptr; },
             [&](int n) {
               const int col = n0 + (n & (MG_BN - 1));
               if (col >= ff) return (const __nv_bfloat16*)nullptr;
               return (n < MG_BN ? wg : wu) + (long long)col * H;
             },
             As, Bs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = warp * 16 + (lane >> 2), c2 = (lane & 3) * 2;
#pragma unroll
  for (int nt = 0; nt < MG_BN / 8; nt++) {
    const int col = n0 + nt * 8 + c2;
    if (col >= ff) continue;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const int r = r0 + half * 8;
      if (r >= rows) continue;
      float v[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (NB == 1) {
          v[j] = gate_act(acc[0][nt][half * 2 + j], act_kind);
          continue;
        }
        const float g = fminf(acc[0][nt][half * 2 + j], limit);
        const float u = fminf(fmaxf(acc[NB - 1][nt][half * 2 + j], -limit), limit);
        v[j] = g * (1.0f / (1.0f + __expf(-alpha * g))) * (u + up_off);
      }
      *reinterpret_cast<__nv_bfloat162*>(act + (long long)(row_first + r) * ff + col) = __floats2bfloat162_rn(v[0], v[1]);
    }
  }
}

__global__ void __launch_bounds__(128)
moe_grouped_down_kernel(const __nv_bfloat16* __restrict__ act, const __nv_bfloat16* __restrict__ w_down,
                        const int* __restrict__ meta, const int* __restrict__ tiles, float* __restrict__ y, int H,
                        int ff) {
  extern __shared__ __align__(16) __nv_bfloat16 mg_smem[];
  __nv_bfloat16* As = mg_smem;
  __nv_bfloat16* Bs = mg_smem + MG_STAGES * MG_BM * MG_LD;
  if ((int)blockIdx.x >= meta[0]) return;
  const int e = tiles[3 * blockIdx.x], row_first = tiles[3 * blockIdx.x + 1], rows = tiles[3 * blockIdx.x + 2];
  const int n0 = blockIdx.y * MG_BN;
  const __nv_bfloat16* wd = w_down + (long long)e * H * ff;
  float acc[1][MG_BN / 8][4];
#pragma unroll
  for (int nt = 0; nt < MG_BN / 8; nt++) acc[0][nt][0] = acc[0][nt][1] = acc[0][nt][2] = acc[0][nt][3] = 0.f;
  mg_tile<1>(acc, ff,
             [&](int r) { return r < rows ? act + (long long)(row_first + r) * ff : nullptr; },
             [&](int n) { return n0 + n < H ? wd + (long long)(n0 + n) * ff : nullptr; }, As, Bs);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = warp * 16 + (lane >> 2), c2 = (lane & 3) * 2;
#pragma unroll
  for (int nt = 0; nt < MG_BN / 8; nt++) {
    const int col = n0 + nt * 8 + c2;
    if (col >= H) continue;
    if (r0 < rows) *reinterpret_cast<float2*>(y + (long long)(row_first + r0) * H + col) = make_float2(acc[0][nt][0], acc[0][nt][1]);
    if (r0 + 8 < rows)
      *reinterpret_cast<float2*>(y + (long long)(row_first + r0 + 8) * H + col) = make_float2(acc[0][nt][2], acc[0][nt][3]);
  }
}

// the kernels read rows in 16-byte pieces and write pairs of columns
MF_API int mf_moe_grouped_ok(int H, int ff, int E) {
  return (H % 8 == 0 && ff % 8 == 0 && E >= 1 && E <= MG_MAX_EXPERTS) ? 1 : 0;
}

// tiles the launches must cover for T tokens with `top` choices each among E experts
MF_API int mf_moe_grouped_max_tiles(int T, int top, int E) { return (T * top + MG_BM - 1) / MG_BM + E; }

MF_API int mf_moe_grouped_up(const void* x, const void* w_gu, const int* row_token, const int* meta, const int* tiles,
                             void* act, int T, int H, int ff, int E, int top, float limit, float alpha, float up_off,
                             int act_kind, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!mf_moe_grouped_ok(H, ff, E)) return MF_ERR_BAD_ARG;
  dim3 grid(mf_moe_grouped_max_tiles(T, top, E), (ff + MG_BN - 1) / MG_BN);
  mf_count(MF_K_MOE_GROUPED);
  const size_t smem = (size_t)MG_STAGES * (MG_BM + 2 * MG_BN) * MG_LD * sizeof(__nv_bfloat16);
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0 || act_kind >= MF_ACT_COUNT) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(moe_grouped_up_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(moe_grouped_up_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  if (act_kind < 0)
    moe_grouped_up_kernel<2><<<grid, 128, smem, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w_gu, row_token,
                                                          meta, tiles, (__nv_bfloat16*)act, H, ff, limit, alpha, up_off,
                                                          act_kind);
  else
    moe_grouped_up_kernel<1><<<grid, 128, smem, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)w_gu, row_token,
                                                          meta, tiles, (__nv_bfloat16*)act, H, ff, limit, alpha, up_off,
                                                          act_kind);
  return (int)cudaGetLastError();
}

MF_API int mf_moe_grouped_down(const void* act, const void* w_down, const int* meta, const int* tiles, float* y, int T,
                               int H, int ff, int E, int top, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (!mf_moe_grouped_ok(H, ff, E)) return MF_ERR_BAD_ARG;
  dim3 grid(mf_moe_grouped_max_tiles(T, top, E), (H + MG_BN - 1) / MG_BN);
  mf_count(MF_K_MOE_GROUPED);
  const size_t smem = (size_t)MG_STAGES * (MG_BM + MG_BN) * MG_LD * sizeof(__nv_bfloat16);
  moe_grouped_down_kernel<<<grid, 128, smem, stream>>>((const __nv_bfloat16*)act, (const __nv_bfloat16*)w_down, meta, tiles,
                                                    y, H, ff);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------ tokens in the order of the rows
// xg[row] = x[row_token[row]], 16 bytes a copy (H a multiple of 8).  A block of several rows: their tokens are looked up
// together, then their pieces are on their way together (12,288 rows of 2,048: a row a block 11.6 us, four 9.6, of which 50 MB of
// writes alone are 7.7 at the copy rate).
constexpr int GATHER_ROWS = 4;
__global__ void __launch_bounds__(256)
moe_gather_rows_kernel(const uint4* x, const int* row_token, uint4* __restrict__ xg, int n_rows, int h8) {
  pdl_launch();
  pdl_wait();
  const int row0 = blockIdx.x * GATHER_ROWS;
  const uint4* src[GATHER_ROWS];
#pragma unroll
  for (int r = 0; r < GATHER_ROWS; r++) src[r] = x + (long long)row_token[min(row0 + r, n_rows - 1)] * h8;
  for (int i = threadIdx.x; i < h8; i += blockDim.x) {
    uint4 v[GATHER_ROWS];
#pragma unroll
    for (int r = 0; r < GATHER_ROWS; r++) v[r] = src[r][i];
#pragma unroll
    for (int r = 0; r < GATHER_ROWS; r++)
      if (row0 + r < n_rows) xg[(long long)(row0 + r) * h8 + i] = v[r];
  }
}

cudaError_t moe_gather_launch(const void* x, const int* row_token, void* xg, int n_rows, int H, cudaStream_t stream) {
  return launch_dep(moe_gather_rows_kernel, dim3((n_rows + GATHER_ROWS - 1) / GATHER_ROWS), dim3(256), 0, stream, (const uint4*)x,
                    row_token, (uint4*)xg, n_rows, H / 8);
}
