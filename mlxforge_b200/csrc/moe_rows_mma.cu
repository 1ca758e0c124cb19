// Experts for few tokens in bfloat16: every chosen expert's matrices are read ONCE, whatever the number of tokens that chose it
// (the block-per-pair kernel of moe.cu reads them once per pair, from L2 where it is lucky).
//
// Every block orders the step's (token, choice) pairs by expert for itself, in the order of the tokens, and cuts an expert's pairs
// into passes of up to NT; a unit is a pass and a slice of 64 of the expert's ff columns.  Persistent blocks, one per SM, walk the
// units.  A producer thread brings, through one ring of 16 KB stages that runs on across units, first the slice's gate and up rows
// (64 of each by 64 columns of H), then the slice's part of the down matrix (128 rows of H by 64 columns).  Eight consumer warps
// multiply with mma.sync.m16n8k16, weights on the M side, tokens on the N side:
//   up     a warp's 16 rows are 8 gate rows and the 8 up rows beside them, so the gate's two factors of a (column, token) meet in one
//          thread; the activation, rounded to bfloat16, goes to shared memory;
//   down   a warp's 16 rows of H times the slice's 64 columns; the 32-bit sums are the slice's share of the pair's result,
//          y [pair, slices, H], which the weighted sum (moe.cu) adds in the order of the slices.
// A column of the products is one token's, so a token's result does not depend on what else is in the step.
// The rows of x of the next unit are copied while this unit multiplies by the down matrix.  Every wait is bounded (codes 81, 82).
//
// What bounds it: the distinct experts' matrices from HBM; a stage is 0.37 us of an SM's share of the copy rate, for which a warp has
// 4 16-byte loads and 4 products a block of 8 tokens.  6 of 64 experts of 768 x 2,048 (the whole mixture, replayed from a graph / launched):
// 8 tokens 116 -> 74 us, of which this kernel 94 -> 65 (about 35 experts, 330 MB); 60 tokens 482 -> 147 us, this kernel 455 -> 120
// (604 MB, 92 us at the copy rate).  With eight stages instead of all that fit (ten) beside the tokens it was 4 us slower.
#include "common.cuh"
#include "tma_host.cuh"

namespace {

constexpr int CW = 8;                                  // consumer warps
constexpr int SLICE = 64;                              // columns of ff in a unit (the slices of moe.cu)
constexpr int STAGE_BYTES = 16384, STAGES_MIN = 8, STAGES_MAX = 11;
constexpr size_t SMEM_MAX = 210 * 1024;               // with the lists below 226 KB
constexpr int HROWS = 128;                             // rows of H in a stage of the down matrix
constexpr int MAX_PAIRS = 512, MAX_EXPERTS = 1024;
constexpr size_t X_BYTES_MAX = 72 * 1024;              // the tokens' rows of a pass
constexpr unsigned WAIT_LIMIT = 1u << 24;

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
__device__ __forceinline__ void mbar_wait(unsigned bar, unsigned parity, int* status, int code) {
  for (unsigned i = 0; i < WAIT_LIMIT; i++) {
    unsigned done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return;
  }
  if (status) atomicExch(status, code);
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int c0, int c1, int c2, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ uint4 lds128(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 bytes into shared memory without a register, zeros where there is nothing to read (bytes = 0)
__device__ __forceinline__ void copy16(unsigned dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(CW * 32) : "memory"); }

struct RowsArgs {
  const __nv_bfloat16* x;
  const int* ids;
  float* y;
  int n_pairs, H, ff, top, n_real, act_kind, slices, n_chunks;      // n_chunks: spans of 64 columns of H
  int stages;
  EpiConst ec;
  int* status;
};

// The pairs ordered by expert (order[]), the passes (expert, first place in order[], pairs) and their number.
struct Lists {
  int ids[MAX_PAIRS], rank[MAX_PAIRS], order[MAX_PAIRS], pass_e[MAX_PAIRS], pass_at[MAX_PAIRS], pass_n[MAX_PAIRS];
  int of_expert[MAX_EXPERTS];      // pairs of an expert, then the place of its first one
  int n_passes;
};

// By one warp, 32 pairs and then 32 experts at a time (378 pairs: about 0.6 us).
template <int NT>
__device__ __forceinline__ void make_lists(const RowsArgs& a, Lists& L, int lane) {
  const unsigned all = 0xffffffffu, below = (1u << lane) - 1;
  for (int e = lane; e < a.n_real; e += 32) L.of_expert[e] = 0;
  __syncwarp();
  for (int i0 = 0; i0 < a.n_pairs; i0 += 32) {
    const int i = i0 + lane;
    const int id = i < a.n_pairs ? L.ids[i] : -1, e = id < a.n_real ? id : -1;        // an identity expert has no matrices
    const unsigned same = __match_any_sync(all, e);
    const int r = __popc(same & below), base = e >= 0 ? L.of_expert[e] : 0;
    __syncwarp();
    if (e >= 0) {
      L.rank[i] = base + r;
      if (r == 0) L.of_expert[e] = base + __popc(same);
    }
    __syncwarp();
  }
  int before = 0, passes = 0;
  for (int e0 = 0; e0 < a.n_real; e0 += 32) {
    const int e = e0 + lane, c = e < a.n_real ? L.of_expert[e] : 0, p = (c + NT - 1) / NT;
    int sum = c | p << 16;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(all, sum, o);
      if (lane >= o) sum += v;
    }
    const int at = before + (sum & 0xffff) - c, first = passes + (sum >> 16) - p;
    if (e < a.n_real) L.of_expert[e] = at;
    for (int q = 0; q < p; q++) {
      L.pass_e[first + q] = e;
      L.pass_at[first + q] = at + q * NT;
      L.pass_n[first + q] = min(NT, c - q * NT);
    }
    const int last = __shfl_sync(all, sum, 31);
    before += last & 0xffff;
    passes += last >> 16;
  }
  __syncwarp();
  for (int i = lane; i < a.n_pairs; i += 32)
    if (L.ids[i] >= 0 && L.ids[i] < a.n_real) L.order[L.of_expert[L.ids[i]] + L.rank[i]] = i;
  if (lane == 0) L.n_passes = passes;
}

// The tokens' rows of a pass into shared memory: [NT][H rounded up to 64], 16-byte pieces of a 128-byte span exchanged like the
// copy engine's 128-byte swizzle does it.  Rows and columns that are not there are zeros.
template <int NT>
__device__ __forceinline__ void load_x(const RowsArgs& a, const Lists& L, int pass, unsigned xs) {
  const int at = L.pass_at[pass], n = L.pass_n[pass], per_row = a.n_chunks * 8;
  for (int i = threadIdx.x; i < NT * per_row; i += CW * 32) {
    const int r = i / per_row, p = i - r * per_row;
    const bool in = r < n && p * 8 < a.H;
    const __nv_bfloat16* src = in ? a.x + (long long)(L.order[at + r] / a.top) * a.H + p * 8 : a.x;
    copy16(xs + (unsigned)(r * per_row + (p ^ (r & 7))) * 16u, src, in ? 16u : 0u);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int NB>
__global__ void __launch_bounds__((CW + 1) * 32, 1)
moe_rows_mma_kernel(const __grid_constant__ CUtensorMap map_gu, const __grid_constant__ CUtensorMap map_down, const RowsArgs a) {
  constexpr int NT = 8 * NB;
  extern __shared__ unsigned char raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  const int STAGES = a.stages;
  const unsigned ring = smem_u32(smem), xs = ring + STAGES * STAGE_BYTES, acts = xs + NT * a.n_chunks * 128;
  const unsigned bars = acts + NT * 128;
  __shared__ Lists L;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool gated = a.act_kind < 0;

  if (threadIdx.x == 0) {
    pdl_launch();
    for (int s = 0; s < STAGES; s++) {
      mbar_init(bars + 8 * s, 1);
      mbar_init(bars + 8 * (STAGES + s), CW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  pdl_wait();
  for (int i = threadIdx.x; i < a.n_pairs; i += blockDim.x) L.ids[i] = a.ids[i];
  __syncthreads();
  if (warp == 0) make_lists<NT>(a, L, lane);
  __syncthreads();
  const int n_units = L.n_passes * a.slices, n_hs = (a.H + HROWS - 1) / HROWS;

  if (warp == CW) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      int s = 0;
      unsigned round = 0;
      for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
        const int pass = u / a.slices, slice = u - pass * a.slices, e = L.pass_e[pass];
        for (int k = 0; k < a.n_chunks + n_hs; k++) {
          const unsigned full = bars + 8 * s, dst = ring + s * STAGE_BYTES;
          if (round > 0) {
            mbar_wait(bars + 8 * (STAGES + s), (round - 1) & 1, a.status, 81);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");       // the readers' loads before the next copy
          }
          if (k < a.n_chunks) {
            mbar_expect_tx(full, gated ? STAGE_BYTES : STAGE_BYTES / 2);         // what lies outside a matrix arrives as zeros
            tma_load_3d(dst, &map_gu, k * 64, slice * SLICE, e * (gated ? 2 : 1), full);
          } else {
            mbar_expect_tx(full, STAGE_BYTES);
            tma_load_3d(dst, &map_down, slice * SLICE, (k - a.n_chunks) * HROWS, e, full);
          }
          if (++s == STAGES) s = 0, round++;
        }
      }
    }
    return;
  }

  // -------------------------------------------------------------- consumers
  const int g = lane >> 2, t = lane & 3;
  if ((int)blockIdx.x < n_units) load_x<NT>(a, L, blockIdx.x / a.slices, xs);
  int s = 0;
  unsigned round = 0;
  for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
    const int pass = u / a.slices, slice = u - pass * a.slices;
    const int at = L.pass_at[pass], n = L.pass_n[pass];
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    consumer_sync();

    // ---- gate and up rows 8 warp .. 8 warp + 7 of the slice; two sums each, of the even and the odd pairs of products
    float acc[NB][2][4];
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[nb][0][j] = acc[nb][1][j] = 0.f;
    for (int k = 0; k < a.n_chunks; k++) {
      uint4 xv[2][NB];
#pragma unroll
      for (int c = 0; c < 2; c++)
#pragma unroll
        for (int nb = 0; nb < NB; nb++)
          xv[c][nb] = lds128(xs + (unsigned)((nb * 8 + g) * a.n_chunks + k) * 128u + ((unsigned)((2 * t + c) ^ g) << 4));
      mbar_wait(bars + 8 * s, round & 1, a.status, 82);
      const unsigned base = ring + s * STAGE_BYTES + (warp * 8 + g) * 128;
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const unsigned piece = (unsigned)((2 * t + c) ^ g) << 4;
        const uint4 w = lds128(base + piece);
        const uint4 v = gated ? lds128(base + SLICE * 128 + piece) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
          mma_bf16(acc[nb][0], w.x, v.x, w.y, v.y, xv[c][nb].x, xv[c][nb].y);
          mma_bf16(acc[nb][1], w.z, v.z, w.w, v.w, xv[c][nb].z, xv[c][nb].w);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (STAGES + s));
      if (++s == STAGES) s = 0, round++;
    }
    // rows beyond ff are zeros, which an input that is not finite turns into NaN
    const bool real = slice * SLICE + warp * 8 + g < a.ff;
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float p = acc[nb][0][j] + acc[nb][1][j], q = acc[nb][0][j + 2] + acc[nb][1][j + 2];
        const float v = real ? gated ? gated_product(p, q, MF_GATE_CLAMPED, a.ec) : gate_act(p, a.act_kind) : 0.f;
        const int tok = nb * 8 + 2 * t + j;
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(acts + tok * 128 + ((unsigned)(warp ^ (tok & 7)) << 4) + g * 2),
                     "h"(__bfloat16_as_ushort(b)) : "memory");
      }
    consumer_sync();

    // ---- the slice's share of the down product; the next unit's tokens on their way meanwhile
    uint4 av[2][NB];
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int nb = 0; nb < NB; nb++) av[c][nb] = lds128(acts + (nb * 8 + g) * 128 + ((unsigned)((2 * t + c) ^ g) << 4));
    if (u + (int)gridDim.x < n_units) load_x<NT>(a, L, (u + gridDim.x) / a.slices, xs);
    float* yo[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int tok = nb * 8 + 2 * t + j;
        yo[nb][j] = tok < n ? a.y + ((long long)L.order[at + tok] * a.slices + slice) * a.H : nullptr;
      }
    for (int hs = 0; hs < n_hs; hs++) {
      float d[NB][4];
#pragma unroll
      for (int nb = 0; nb < NB; nb++) d[nb][0] = d[nb][1] = d[nb][2] = d[nb][3] = 0.f;
      mbar_wait(bars + 8 * s, round & 1, a.status, 82);
      const unsigned base = ring + s * STAGE_BYTES + (warp * 16 + g) * 128;
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const unsigned piece = (unsigned)((2 * t + c) ^ g) << 4;
        const uint4 w = lds128(base + piece), v = lds128(base + 1024 + piece);
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
          mma_bf16(d[nb], w.x, v.x, w.y, v.y, av[c][nb].x, av[c][nb].y);
          mma_bf16(d[nb], w.z, v.z, w.w, v.w, av[c][nb].z, av[c][nb].w);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + 8 * (STAGES + s));
      if (++s == STAGES) s = 0, round++;
      const int h = hs * HROWS + warp * 16 + g;
#pragma unroll
      for (int nb = 0; nb < NB; nb++)
#pragma unroll
        for (int j = 0; j < 2; j++)
          if (yo[nb][j]) {
            if (h < a.H) yo[nb][j][h] = d[nb][j];
            if (h + 8 < a.H) yo[nb][j][h + 8] = d[nb][j + 2];
          }
    }
    // the next unit writes `acts` behind the barrier after its copies: every warp has read its part by then
  }
}

// [layers][rows][cols] row-major bfloat16 with boxes of box_layers x box_rows x 64 columns, 128-byte swizzle
int map_3d(const void* ptr, long long cols, long long rows, long long layers, int box_rows, int box_layers, CUtensorMap* out) {
  tma_host::EncodeTiled enc = tma_host::encoder();
  if (!enc) return MF_ERR_BAD_ARG;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)layers};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)cols * rows * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)box_layers};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 20000 + (int)r;
}

template <int NB>
int launch(const void* w_gu, const void* w_down, RowsArgs a, cudaStream_t stream) {
  const bool gated = a.act_kind < 0;
  CUtensorMap mg, md;
  int rc = map_3d(w_gu, a.H, a.ff, (long long)a.n_real * (gated ? 2 : 1), SLICE, gated ? 2 : 1, &mg);
  if (rc) return rc;
  rc = map_3d(w_down, a.ff, a.H, a.n_real, HROWS, 1, &md);
  if (rc) return rc;
  // as many stages as there is room for beside the tokens: an SM has to keep most of its shared memory on the way
  const size_t rest = 1024 + (size_t)NB * 8 * (a.n_chunks + 1) * 128 + 16 * STAGES_MAX;
  const size_t room = (SMEM_MAX - rest) / STAGE_BYTES;
  a.stages = room < STAGES_MAX ? (int)room : STAGES_MAX;
  if (a.stages < STAGES_MIN) return MF_ERR_BAD_ARG;
  const size_t smem = rest + (size_t)a.stages * STAGE_BYTES;
  static DeviceOnce once;
  const int dev = mf_current_device(), n_sms = mf_sm_count();
  if (dev < 0 || n_sms <= 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(moe_rows_mma_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  const long long most_units = (long long)a.n_pairs * a.slices;
  mf_count(MF_K_MOE_ROWS);
  mf_count(MF_K_MOE_ROWS_MMA);
  return (int)launch_dep(moe_rows_mma_kernel<NB>, dim3((unsigned)(most_units < n_sms ? most_units : n_sms)),
                         dim3((CW + 1) * 32), smem, stream, mg, md, a);
}

}  // namespace

// Tokens of a pass for rows of H: 16, 8 (rows so wide that 16 of them leave no room beside the ring), or 0 (neither fits).
static int rows_mma_tokens(int H) {
  const size_t row = (size_t)((H + 63) / 64) * 128;
  return 16 * row <= X_BYTES_MAX ? 16 : 8 * row <= X_BYTES_MAX ? 8 : 0;
}

bool moe_rows_mma_ok(const void* x, const void* w_gu, const void* w_down, int T, int H, int ff, int top, int n_real) {
  return n_real > 0 && H % 8 == 0 && ff % 8 == 0 && (long long)T * top <= MAX_PAIRS && rows_mma_tokens(H) > 0 &&
         !(((uintptr_t)x | (uintptr_t)w_gu | (uintptr_t)w_down) & 15) && n_real <= MAX_EXPERTS;
}

int moe_rows_mma(const void* x, const void* w_gu, const void* w_down, const int* ids, float* y, int T, int H, int ff, int top,
                 const EpiConst& ec, int n_real, int act_kind, int* status, cudaStream_t stream) {
  const RowsArgs a{(const __nv_bfloat16*)x, ids, y, T * top, H, ff, top, n_real, act_kind, (ff + SLICE - 1) / SLICE,
                   (H + 63) / 64, 0, ec, status};
  // eight tokens or fewer never fill more than half of a wide pass
  return T > 8 && rows_mma_tokens(H) == 16 ? launch<2>(w_gu, w_down, a, stream) : launch<1>(w_gu, w_down, a, stream);
}
