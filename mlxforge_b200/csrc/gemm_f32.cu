// C[M,N] = A[M,K] * W[N,K]^T in IEEE float32 on the CUDA cores: no tensor
// cores, no TF32.  This is the matrix product of the 32-bit model path (the
// reference has no such path; its products are fp16 `mx::matmul`,
// src/model/decoder_model.cpp:174-192).  Each output element is four serial FMA
// chains, chain g over the k with k / 16 = g modulo 4 in increasing order, added
// as (c0 + c1) + (c2 + c3): K alone decides the order, so a value does not depend on M, on the
// tile it falls in or on what else is in the batch.
//
// Four groups of threads work on a block's tile of results, a chain each: a group alone (one warp per scheduler) leaves
// the FMA pipe idle while its operands come from shared memory.  A group's next 16 k are on their way to registers while it
// multiplies 16.  Two bounds decide a thread's tile: a lane gets at most four bytes a cycle from shared memory (8 x 8
// results read 16 numbers for 64 multiplications, 4 x 4 read 8 for 16), and the scheduler issues one instruction a cycle
// (two rows in one packed multiplication leave it room for the loads: 134 -> 111 us at 300 x 3072 x 2048).
// Measured (rows x N x K, before: 64 x 64 tiles of 4 x 4 results a thread, one chain): 8 x 3072 x 2048 155 -> 28 us,
// 64 x 3072 x 2048 158 -> 49, 300 x 3072 x 2048 244 -> 111, 2048 x 3072 x 2048 1202 -> 580 (44 TFLOP/s); the shorter chains
// halve the error against 64 bits (8.1e-7 -> 4.1e-7 at K 2048).  16 x 8 results a thread, which read a quarter less, take as long as
// 8 x 8 (114 and 112 us at 300 x 3072 x 2048), so shared memory is not what is left; single multiplications 129.
#include "common.cuh"

namespace {
constexpr int BK = 16;
constexpr int GROUPS = 4;

// A tile in shared memory: [k][rows of A, then rows of W], padded to whole 32.  Row r of k stands at r ^ (k / 4 % 4) * 8: a
// warp loads 16 neighbouring k of eight rows at a time (whole 64-byte pieces of the matrices) and stores them without two in
// a bank.
constexpr int tile_ld(int bm, int bn) { return (bm + bn + 31) / 32 * 32; }
constexpr int tile_floats(int bm, int bn) { return BK * tile_ld(bm, bn); }
constexpr int threads_of(int bm, int bn, int tm, int tn) { return (bm / tm) * (bn / tn); }      // of a group: one per tile of results

// VEC: rows are whole 16-byte pieces (K a multiple of 4, aligned operands)
template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(threads_of(BM, BN, TM, TN) * GROUPS)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                int accumulate) {
  constexpr int TG = threads_of(BM, BN, TM, TN);
  constexpr int LD = tile_ld(BM, BN), TILE = tile_floats(BM, BN);
  constexpr int PIECES = (BM + BN) * (BK / 4);         // 4 neighbouring k of a row
  constexpr int PER = (PIECES + TG - 1) / TG;
  extern __shared__ __align__(16) float sm[];          // [GROUPS][2][TILE]; at the end the groups' results
  const int group = threadIdx.x / TG, tid = threadIdx.x % TG;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float* mine = sm + group * 2 * TILE;
  float4 next[PER];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int i = tid + p * TG, row = i / 4, k = k0 + i % 4 * 4;
      const bool is_a = row < BM;
      const int g = is_a ? m0 + row : n0 + row - BM;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < PIECES && g < (is_a ? M : N) && k < K) {
        const float* src = (is_a ? A : W) + (long long)g * K + k;
        if (VEC) {
          x = *reinterpret_cast<const float4*>(src);
        } else {
          x.x = src[0];
          if (k + 1 < K) x.y = src[1];
          if (k + 2 < K) x.z = src[2];
          if (k + 3 < K) x.w = src[3];
        }
      }
      next[p] = x;
    }
  };
  auto place = [&](int buf) {
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int i = tid + p * TG, row = i / 4, kq = i % 4;
      if (i >= PIECES) continue;
      float* dst = mine + buf * TILE + kq * 4 * LD + (row ^ kq * 8);
      dst[0] = next[p].x;
      dst[LD] = next[p].y;
      dst[2 * LD] = next[p].z;
      dst[3 * LD] = next[p].w;
    }
  };
  auto group_barrier = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "n"(TG) : "memory"); };
  // the thread's rows: four neighbours and further fours BM / (TM / 4) apart; its columns likewise
  constexpr int RSTEP = BM / (TM / 4), CSTEP = TN >= 4 ? BN / (TN / 4) : BN;
  const int tr = tid / (BN / TN) * 4, tc = tid % (BN / TN) * (TN < 4 ? TN : 4);
  f32x2 acc[TM / 2][TN];                               // two neighbouring rows a register pair
#pragma unroll
  for (int i = 0; i < TM / 2; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = pack2(0.f, 0.f);
  int k0 = group * BK, buf = 0;
  if (k0 < K) {
    fetch(k0);
    place(0);
  }
  group_barrier();
  for (; k0 < K; k0 += GROUPS * BK, buf ^= 1) {
    const bool more = k0 + GROUPS * BK < K;
    if (more) fetch(k0 + GROUPS * BK);
    const float* tile = mine + buf * TILE;
#pragma unroll
    for (int k = 0; k < BK; k++) {
      const float* row = tile + k * LD;
      const int turn = k / 4 * 8;
      alignas(16) f32x2 a[TM / 2];
      alignas(16) float b[TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4)
        *reinterpret_cast<ulonglong2*>(a + i / 2) =
            *reinterpret_cast<const ulonglong2*>(row + ((tr + i / 4 * RSTEP) ^ turn));
      if constexpr (TN >= 4) {
#pragma unroll
        for (int j = 0; j < TN; j += 4)
          *reinterpret_cast<float4*>(b + j) = *reinterpret_cast<const float4*>(row + ((BM + tc + j / 4 * CSTEP) ^ turn));
      } else {
        b[0] = row[(BM + tc) ^ turn];
      }
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const f32x2 bb = pack2(b[j], b[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; i++) acc[i][j] = fma2(a[i], bb, acc[i][j]);
      }
    }
    // the other buffer was read last one turn ago, before the barrier that ended it
    if (more) place(buf ^ 1);
    group_barrier();
  }
  // the four chains meet: a group's results stand [result][thread], one group after another
  __syncthreads();
  float* meet = sm;
#pragma unroll
  for (int i = 0; i < TM / 2; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const float2 v = unpack2(acc[i][j]);
      meet[((group * TM + 2 * i) * TN + j) * TG + tid] = v.x;
      meet[((group * TM + 2 * i + 1) * TN + j) * TG + tid] = v.y;
    }
  __syncthreads();
  constexpr int SHARE = TM * TN / GROUPS;              // results of a thread's tile that this group finishes
#pragma unroll
  for (int s = 0; s < SHARE; s++) {
    const int e = group * SHARE + s, i = e / TN, j = e % TN;
    auto chain = [&](int g) { return meet[(g * TM * TN + e) * TG + tid]; };
    const float sum = (chain(0) + chain(1)) + (chain(2) + chain(3));
    const int gm = m0 + tr + (i & 3) + (i >> 2) * RSTEP, gn = n0 + tc + (j & 3) + (j >> 2) * CSTEP;
    if (gm < M && gn < N) {
      float* c = C + (long long)gm * N + gn;
      *c = accumulate ? (*c + sum) : sum;
    }
  }
}

template <int BM, int BN, int TM, int TN, bool VEC>
int launch_one(const float* A, const float* W, float* C, int M, int N, int K, int accumulate, cudaStream_t stream) {
  constexpr int floats = 2 * tile_floats(BM, BN) > BM * BN ? 2 * tile_floats(BM, BN) : BM * BN;
  constexpr size_t smem = (size_t)GROUPS * floats * sizeof(float);
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return MF_ERR_BAD_ARG;
  mf_count(MF_K_GEMM_F32);
  gemm_f32_kernel<BM, BN, TM, TN, VEC><<<grid, threads_of(BM, BN, TM, TN) * GROUPS, smem, stream>>>(A, W, C, M, N, K, accumulate);
  return (int)cudaGetLastError();
}

template <int BM, int BN, int TM, int TN>
int launch(const float* A, const float* W, float* C, int M, int N, int K, int accumulate, cudaStream_t stream) {
  const bool vec = K % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
  return vec ? launch_one<BM, BN, TM, TN, true>(A, W, C, M, N, K, accumulate, stream)
             : launch_one<BM, BN, TM, TN, false>(A, W, C, M, N, K, accumulate, stream);
}
}  // namespace

MF_API int mf_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int accumulate,
                       cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return MF_ERR_BAD_ARG;
  if (M <= 16) return launch<16, 32, 4, 1>(A, W, C, M, N, K, accumulate, stream);
  // The tile whose blocks go around the SMs in the least time: rounds of blocks times a block's time, which was measured at K 2,048
  // for at most one block an SM (us); every tile adds an element's terms in the same order.  More blocks of a small tile fit an SM at once, which
  // the rounds leave out; no M of 17 to 2,048 at eight widths is slower by more than 2 % than with the one tile that all had before.
  const int sms = mf_sm_count();
  if (sms <= 0) return MF_ERR_BAD_ARG;
  auto time = [&](int bm, int bn, float block) {
    // the tallest operand that the grid's second dimension holds is 65535 tiles of 64 rows
    if ((M + bm - 1) / bm > 65535) return INFINITY;
    const long long blocks = (long long)((N + bn - 1) / bn) * ((M + bm - 1) / bm);
    return (float)((blocks + sms - 1) / sms) * block;
  };
  const float t[4] = {time(64, 128, 107.f), time(48, 128, 88.f), time(64, 64, 70.f), time(32, 64, 45.f)};
  if (t[3] < t[0] && t[3] <= t[1] && t[3] <= t[2]) return launch<32, 64, 4, 4>(A, W, C, M, N, K, accumulate, stream);
  if (t[2] < t[0] && t[2] <= t[1]) return launch<64, 64, 8, 8>(A, W, C, M, N, K, accumulate, stream);
  if (t[1] < t[0]) return launch<48, 128, 12, 8>(A, W, C, M, N, K, accumulate, stream);
  return launch<64, 128, 8, 8>(A, W, C, M, N, K, accumulate, stream);
}
