// Experts for many tokens on the 5th-generation tensor cores: the two products over the pairs ordered by expert
// (moe_grouped.cu), with the WEIGHTS on the M side of tcgen05.mma.  A unit is 128 rows of an expert's matrix times up to 256 of
// its pairs, so that an expert with 200 pairs reads its matrices once and multiplies hardly more than it has (N is the pairs
// rounded up to 16), where tiles with the pairs on the M side read them once per 64 or 128 pairs.
//
//   up     D_gate, D_up [128 rows of ff, pairs] over H, both from one tile of the tokens; the clamped gate (or an ungated
//          expert's activation) on the 32-bit sums in the epilogue, act [pair, ff] in bfloat16;
//   down   D [128 rows of H, pairs] over ff; y [pair, H] in bfloat16 or 32-bit.
//
// Persistent blocks, one per SM, walk the units (the 128-row slices of one expert's pairs beside one another, so that the
// pairs' rows come from L2): warp 0 issues the tensor copies of 64-wide K steps into a ring, warp 1 the products, warps 2-9
// are the epilogue (a warp may read the tensor memory lanes of its number modulo 4; two share a quarter and take turns by 16
// columns).  The gated product's two accumulators fill the tensor memory; the others alternate between two.
// Rows of a tile beyond the expert's matrix or the pairs' range are other valid memory or zeros; their results are not stored.
// Every wait is bounded (codes 71-74 in `status`), and the tensor memory is freed in every case.
//
// What bounds it: 64 experts of 768 x 2,048 are 604 MB, 92 us at the copy bandwidth, and 12,288 pairs 70 us of products.
// The whole mixture for 2,048 tokens (6 of 64 experts): 225 -> 190 us against the library's grouped product with its own activation
// pass (up 95, down 48; the gated product's units go 2.6 times around the SMs), for 64 tokens 184 -> 137, for 513 tokens of 32
// experts of 512 x 1,024 110 -> 62.  Sending for the weights eight K steps ahead into L2 was slower (up 110 us, sixteen ahead 133).
#include "common.cuh"
#include "tma_host.cuh"

namespace {

constexpr int MT = 128, NT = 256, BK = 64, BOX = 64;         // rows of a unit; its most pairs; a K step; pairs of one copy
constexpr unsigned WAIT_LIMIT = 1u << 26;
constexpr int A_BYTES = MT * BK * 2, B_BYTES = NT * BK * 2;
enum { GATED = 0, PLAIN = 1, DOWN = 2, DOWN_F32 = 3 };
template <int MODE> struct Ring {
  static constexpr int A = MODE == GATED ? 2 : 1;
  static constexpr int STAGES = MODE == GATED ? 3 : 4;
  static constexpr int STAGE_BYTES = A * A_BYTES + B_BYTES;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + (2 * STAGES + 4) * 8 + 16 + 1024;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
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
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int c0, int c1, unsigned bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// K-major operand tile, rows of 64 bfloat16, 128-byte swizzle: groups of 8 rows are 1024 bytes apart
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr >> 4) & 0x3FFF);
  d |= (unsigned long long)1 << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;
  d |= (unsigned long long)1 << 46;
  d |= (unsigned long long)2 << 61;
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
__device__ __forceinline__ void umma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
  unsigned r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

struct Unit {
  int expert, row0, rows, slice;
};
__device__ __forceinline__ Unit unit_at(int u, int slices, const int* __restrict__ tiles) {
  const int b = u / slices;
  return Unit{tiles[3 * b], tiles[3 * b + 1], tiles[3 * b + 2], u - b * slices};
}

// rows_w: rows of an expert's matrix that a unit's slices cut up (ff, or H for the second product); stride_w: rows from an
// expert's matrix to the next (the gate's rows, then the up matrix's, are one)
template <int MODE>
__global__ void __launch_bounds__(320, 1)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_b,
              const int* __restrict__ meta, const int* __restrict__ tiles, void* __restrict__ out_, int rows_w,
              int stride_w, int K, int act_kind, EpiConst ec, int* __restrict__ status) {
  using R = Ring<MODE>;
  constexpr int STAGES = R::STAGES;
  extern __shared__ unsigned char raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + STAGES * R::STAGE_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * STAGES + 4);
  const unsigned smem_u = smem_u32(smem), bars_u = smem_u32(bars);
  const unsigned full0 = bars_u, empty0 = bars_u + 8 * STAGES;
  const unsigned acc_full0 = bars_u + 16 * STAGES, acc_empty0 = acc_full0 + 16;
  constexpr int ACCS = MODE == GATED ? 1 : 2;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slices = (rows_w + MT - 1) / MT, n_units = meta[0] * slices;
  const int n_kt = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(acc_full0 + 8 * a, 1);
      mbar_init(acc_empty0 + 8 * a, 8);      // one arrive per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      unsigned it = 0;
      for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
        const Unit w = unit_at(u, slices, tiles);
        const int wr = w.expert * stride_w + w.slice * MT, boxes = max(1, (w.rows + BOX - 1) / BOX);
        for (int kt = 0; kt < n_kt; kt++, it++) {
          const unsigned s = it % STAGES, round = it / STAGES;
          if (round > 0) mbar_wait(empty0 + 8 * s, (round - 1) & 1, status, 71);
          const unsigned full = full0 + 8 * s, at = smem_u + s * R::STAGE_BYTES;
          mbar_expect_tx(full, R::A * A_BYTES + boxes * (BOX * BK * 2));
          tma_load_2d(at, &map_w, kt * BK, wr, full);
          if (MODE == GATED) tma_load_2d(at + A_BYTES, &map_w, kt * BK, wr + rows_w, full);
          for (int b = 0; b < boxes; b++)
            tma_load_2d(at + R::A * A_BYTES + b * (BOX * BK * 2), &map_b, kt * BK, w.row0 + b * BOX, full);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ issuer
    if (lane == 0) {
      unsigned it = 0, i = 0;
      for (int u = blockIdx.x; u < n_units; u += gridDim.x, i++) {
        const Unit w = unit_at(u, slices, tiles);
        const unsigned n16 = (unsigned)max(16, (w.rows + 15) / 16 * 16);        // a cut may leave a tile empty
        // D float32, A and B bfloat16, both K-major; N >> 3 at bit 17, M >> 4 at bit 24
        const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n16 >> 3) << 17) | ((unsigned)(MT >> 4) << 24);
        const unsigned acc = i % ACCS, use = i / ACCS;
        if (use > 0) {
          mbar_wait(acc_empty0 + 8 * acc, (use - 1) & 1, status, 74);     // the epilogue has drained it
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        }
        const unsigned tmem_c = tmem_base + acc * NT;
        for (int kt = 0; kt < n_kt; kt++, it++) {
          const unsigned s = it % STAGES, round = it / STAGES;
          mbar_wait(full0 + 8 * s, round & 1, status, 72);
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const unsigned a_addr = smem_u + s * R::STAGE_BYTES, b_addr = a_addr + R::A * A_BYTES;
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; k4++) {
            const unsigned go_on = (kt > 0 || k4 > 0) ? 1u : 0u;
            umma(tmem_c, smem_desc(a_addr + k4 * 32), smem_desc(b_addr + k4 * 32), idesc, go_on);
            if (MODE == GATED)
              umma(tmem_c + NT, smem_desc(a_addr + A_BYTES + k4 * 32), smem_desc(b_addr + k4 * 32), idesc, go_on);
          }
          umma_commit(empty0 + 8 * s);
        }
        umma_commit(acc_full0 + 8 * acc);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int lg = warp & 3, half = (warp - 2) >> 2;
    const bool odd = lane & 1;
    unsigned i = 0;
    for (int u = blockIdx.x; u < n_units; u += gridDim.x, i++) {
      const Unit w = unit_at(u, slices, tiles);
      const unsigned acc = i % ACCS, use = i / ACCS;
      const int f = w.slice * MT + lg * 32 + lane;                // this lane's row of the matrix: a column of `out`
      mbar_wait(acc_full0 + 8 * acc, use & 1, status, 73);
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const unsigned taddr = tmem_base + ((unsigned)(lg * 32) << 16) + acc * NT;
      for (int c = half * 16; c < w.rows; c += 32) {
        float v[16];
        tmem_ld16(taddr + c, v);
        if (MODE == GATED) {
          float up[16];
          tmem_ld16(taddr + NT + c, up);
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = gated_product<true>(v[j], up[j], MF_GATE_CLAMPED, ec);
        } else if (MODE == PLAIN) {
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = gate_act(v[j], act_kind);
        }
        if (MODE == DOWN_F32) {
          float* out = reinterpret_cast<float*>(out_);
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (c + j < w.rows && f < rows_w) out[(long long)(w.row0 + c + j) * rows_w + f] = v[j];
          continue;
        }
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(out_);
        // two neighbouring lanes trade, so that each stores two neighbouring columns of one pair's row
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float got = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
          const __nv_bfloat162 o = odd ? __floats2bfloat162_rn(got, v[j + 1]) : __floats2bfloat162_rn(v[j], got);
          const int row = c + j + (odd ? 1 : 0);
          if (row < w.rows && f < rows_w)
            *reinterpret_cast<__nv_bfloat162*>(out + (long long)(w.row0 + row) * rows_w + (f & ~1)) = o;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_empty0 + 8 * acc) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
  }
}

template <int MODE>
int launch(const void* w, long long w_rows, const void* b, int n_pairs, const int* meta, const int* tiles, void* out,
           int rows_w, int stride_w, int K, int act_kind, const EpiConst& ec, int max_units, int* status,
           cudaStream_t stream) {
  CUtensorMap mw, mb;
  int rc = tma_host::bf16_map(w, w_rows, K, MT, BK, &mw);
  if (rc) return rc;
  rc = tma_host::bf16_map(b, n_pairs, K, BOX, BK, &mb);
  if (rc) return rc;
  static DeviceOnce once;
  const int dev = mf_current_device(), n_sms = mf_sm_count();
  if (dev < 0 || n_sms <= 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(moe_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Ring<MODE>::SMEM);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  mf_count(MF_K_MOE_GROUPED);
  mf_count(MF_K_MOE_GROUPED_TC);
  moe_tc_kernel<MODE><<<max_units < n_sms ? max_units : n_sms, 320, Ring<MODE>::SMEM, stream>>>(
      mw, mb, meta, tiles, out, rows_w, stride_w, K, act_kind, ec, status);
  return (int)cudaGetLastError();
}

}  // namespace

cudaError_t moe_gather_launch(const void* x, const int* row_token, void* xg, int n_rows, int H, cudaStream_t stream);

// Pairs of a unit: what mf_moe_sort cuts an expert's rows into for these products.
MF_API int mf_moe_tc_rows() { return NT; }

static bool tc_ok(const void* w, const void* b, const void* out, int H, int ff, int E, long long w_rows) {
  return !(((uintptr_t)w | (uintptr_t)b) & 15) && !((uintptr_t)out & 3) && H % 8 == 0 && ff % 8 == 0 && H > 0 && ff > 0 && E > 0 &&
         w_rows <= 0x7fffffff;
}

// x [T, H]; xg [n_pairs, H]: scratch, the tokens in the order of the pairs (row_token); w_gu [E, 2, ff, H] (act_kind < 0: the clamped gate) or [E, 1, ff, H];
// tiles and meta from mf_moe_sort with tile rows of mf_moe_tc_rows(); act [n_pairs, ff].
MF_API int mf_moe_tc_up(const void* x, const int* row_token, void* xg, const void* w_gu, const int* meta, const int* tiles, void* act, int n_pairs, int H,
                        int ff, int E, float limit, float alpha, float up_off, int act_kind, int* status,
                        cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  const int parts = act_kind < 0 ? 2 : 1;
  if (!tc_ok(w_gu, xg, act, H, ff, E, (long long)E * parts * ff) || act_kind >= MF_ACT_COUNT) return MF_ERR_BAD_ARG;
  const EpiConst ec{limit, alpha, up_off, 0.f};
  const int units = (n_pairs / NT + E) * ((ff + MT - 1) / MT);
  const cudaError_t e = moe_gather_launch(x, row_token, xg, n_pairs, H, stream);
  if (e != cudaSuccess) return (int)e;
  if (act_kind < 0)
    return launch<GATED>(w_gu, (long long)E * 2 * ff, xg, n_pairs, meta, tiles, act, ff, 2 * ff, H, act_kind, ec, units, status, stream);
  return launch<PLAIN>(w_gu, (long long)E * ff, xg, n_pairs, meta, tiles, act, ff, ff, H, act_kind, ec, units, status, stream);
}

// y [n_pairs, H] in y_dtype = act w_down[e]^T, w_down [E, H, ff].
MF_API int mf_moe_tc_down(const void* act, const void* w_down, const int* meta, const int* tiles, void* y, int y_dtype,
                          int n_pairs, int H, int ff, int E, int* status, cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (!tc_ok(w_down, act, y, H, ff, E, (long long)E * H)) return MF_ERR_BAD_ARG;
  const int units = (n_pairs / NT + E) * ((H + MT - 1) / MT);
  if (y_dtype == MF_F32)
    return launch<DOWN_F32>(w_down, (long long)E * H, act, n_pairs, meta, tiles, y, H, H, ff, -1, EpiConst{}, units, status, stream);
  if (y_dtype != MF_BF16) return MF_ERR_BAD_DTYPE;
  return launch<DOWN>(w_down, (long long)E * H, act, n_pairs, meta, tiles, y, H, H, ff, -1, EpiConst{}, units, status, stream);
}
