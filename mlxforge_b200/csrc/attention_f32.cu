// Causal grouped-query attention over the paged cache in IEEE float32, with the options of attention_generic.cu (window,
// kept first keys, sink, output gate, soft cap, values of their own width or inside the keys), a block per tile of queries.
//
// A tile's rows are (token, query head of one KV head), so that one copy of the keys serves all of them; 64 keys at a time,
// tiles at multiples of 64 of the sequence.  Per tile of keys: S = Q K^T and O += P V as products of 4 x 8 results a thread
// over operands in shared memory, the softmax between them in registers (a row's scores lie in 8 neighbouring lanes).
// Decoding takes tiles of 16 rows, so that few rows do not pay for 64; a row's sums have one order in either, so they do not
// depend on what else is in the step.
//
// A key's values meet a weight of zero in the rows of a tile that do not see it, and one that is not finite makes them NaN: rows
// whose result is not finite are worked out again over their own keys (row_again). Telling such values apart in the loop over
// the tiles instead (while they are copied, before a tile's product, behind it) cost the finite ones 1 to 27 %.
//
// The block per (token, head) of attention_generic.cu read every key row again for each of them, a lane a row of its own.
// The layers around the two (projections included; us before -> now): 32 / 8 heads of 64, 300 tokens 964 -> 251; a latent of 192 + 32
// under 16 heads, 150 tokens behind 300 keys 619 -> 334 with rows of keys looked up once a tile, values on their way while the
// scores are made and tiles of 32 and 16 rows (8 tokens behind 1,000 keys 420 -> 261; 32 / 8 heads of 128 514 -> 268).
// That kernel stays for bfloat16 at sizes the tensor-core kernels do not take and for rows that are no whole 16-byte pieces.
#include "common.cuh"

namespace {
constexpr int KT = 64;                   // keys of a tile

struct F32Args {
  const float *q, *k_pool, *v_pool;
  float* out;
  const int *q_start, *q_len, *ctx_len;
  PagedView pv;
  int n_heads, rep, tokens;              // heads of a KV head; tokens of a tile
  float scale;
  int window, vd, v_ld, keep_first;
  const float *sink, *gate;
  long long gate_ld;
  float softcap;
};

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// whether the query at `pos` (-1: none) sees `key`
__device__ __forceinline__ bool sees(const F32Args& a, int pos, int key) {
  return key <= pos && (a.window <= 0 || pos - key < a.window || key < a.keep_first);
}

// N floats in pieces of up to four from p on, pieces `step` apart
template <int N>
__device__ __forceinline__ void get(float (&x)[N], const float* p, int step) {
  if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    x[0] = t.x; x[1] = t.y;
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 t = load4(p + i / 4 * step);
      x[i] = t.x; x[i + 1] = t.y; x[i + 2] = t.z; x[i + 3] = t.w;
    }
  }
}

// A row's results again, for columns c0 + (j & 3) + (j >> 2) * CSTEP of VC pieces of 64: the sums of the kernel below in their order,
// over the keys that the row sees alone.  For rows whose result is not finite: the kernel multiplies a key's values with a
// weight of zero for the rows of a tile that do not see it, which lets a value that is not finite into them.
template <int VC, int CPT, int CSTEP>
__device__ __noinline__ void row_again(const F32Args& a, int seq, int t, int h, int pos, int c0, float inv) {
  const int hd = a.pv.head_dim, kvh = h / a.rep;
  const int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0, keep = a.window > 0 ? min(a.keep_first, lo) : 0;
  const float* q = a.q + ((long long)t * a.n_heads + h) * hd;
  float m = a.sink ? a.sink[h] : -INFINITY, p[KT], o[VC * CPT];
#pragma unroll
  for (int i = 0; i < VC * CPT; i++) o[i] = 0.f;
  auto column = [&](int i) { return i / CPT * 64 + c0 + (i % CPT & 3) + (i % CPT >> 2) * CSTEP; };
  const int first_win = lo / KT * KT;
#pragma unroll 1
  for (int k0 = keep > 0 ? 0 : first_win; k0 <= pos; k0 += KT) {
    if (k0 < first_win && k0 >= keep) {
      k0 = first_win - KT;
      continue;
    }
    float top = m;
#pragma unroll 1
    for (int j = 0; j < KT; j++) {
      p[j] = -INFINITY;
      if (!sees(a, pos, k0 + j)) continue;
      const float* k = a.k_pool + paged_offset(a.pv, seq, k0 + j, kvh);
      float s = 0.f;
#pragma unroll 1
      for (int d0 = 0; d0 < hd; d0 += 16) {
        float part = 0.f;
#pragma unroll 1
        for (int d = d0; d < min(hd, d0 + 16); d++) part = fmaf(q[d], k[d], part);
        s += part;
      }
      s = __fmul_rn(s, a.scale);
      if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
      p[j] = s;
      top = fmaxf(top, s);
    }
    const float fade = m == -INFINITY ? 0.f : expf(m - top);
    m = top;
#pragma unroll
    for (int i = 0; i < VC * CPT; i++) o[i] *= fade;
#pragma unroll 1
    for (int j0 = 0; j0 < KT; j0 += 16) {
      float part[VC * CPT];
#pragma unroll
      for (int i = 0; i < VC * CPT; i++) part[i] = 0.f;
#pragma unroll 1
      for (int j = j0; j < j0 + 16; j++) {
        if (!sees(a, pos, k0 + j)) continue;
        const float w = p[j] == -INFINITY ? 0.f : expf(p[j] - top);
        const float* v = a.v_pool + paged_offset(a.pv, seq, k0 + j, kvh) / hd * a.v_ld;
#pragma unroll
        for (int i = 0; i < VC * CPT; i++)
          if (column(i) < a.vd) part[i] = fmaf(w, v[column(i)], part[i]);
      }
#pragma unroll
      for (int i = 0; i < VC * CPT; i++) o[i] += part[i];
    }
  }
  float* dst = a.out + ((long long)t * a.n_heads + h) * a.vd;
  const float* gate = a.gate ? a.gate + (long long)t * a.gate_ld + (long long)h * a.vd : nullptr;
#pragma unroll
  for (int i = 0; i < VC * CPT; i++) {
    const int c = column(i);
    if (c < a.vd) dst[c] = gate ? o[i] * inv * (1.0f / (1.0f + expf(-gate[c]))) : o[i] * inv;
  }
}

// RT rows, values in VC pieces of 64 columns.  Queries and keys stand in shared memory transposed, [channel][row], row r of
// channel d at r ^ (d / 4 % 4) * 8: a warp reads 64 bytes of eight rows at a time and stores them without two in a bank.
template <int RT, int VC>
__global__ void __launch_bounds__(128)
attention_f32_kernel(const F32Args a) {
  constexpr int CG = RT == 64 ? 8 : 16;            // lanes that share rows
  constexpr int RPT = RT * CG / 128, CPT = KT / CG;            // a thread's rows; its columns of 64
  constexpr int CSTEP = KT / (CPT > 4 ? CPT / 4 : 1);          // between its two groups of four columns
  constexpr int VW = VC * 64, RP = RT + 4;
  const int hd = a.pv.head_dim, dp = (hd + 15) / 16 * 16;
  extern __shared__ __align__(16) float sm[];
  float* qt = sm;                                  // [dp][RT]
  float* kt = qt + dp * RT;                        // [dp][KT]
  float* vs = kt + dp * KT;                        // [KT][VW]
  float* pt = vs + KT * VW;                        // [KT][RP]
  const int seq = blockIdx.z, kvh = blockIdx.y, tid = threadIdx.x;
  const int n = a.q_len[seq];
  const int tile = (n + a.tokens - 1) / a.tokens - 1 - blockIdx.x;       // the tiles with the most keys first
  if (tile < 0) return;
  const int q0 = tile * a.tokens, nq = min(a.tokens, n - q0);
  const int t0 = a.q_start[seq] + q0, pos0 = a.ctx_len[seq] - n + q0;    // token and position of the tile's first row
  const int rows = nq * a.rep;
  const int last = pos0 + nq - 1;
  const int lo = a.window > 0 ? max(0, pos0 - a.window + 1) : 0;         // first key in any row's window
  const int keep = a.window > 0 ? min(a.keep_first, lo) : 0;             // kept keys before it

  // queries, transposed; rows and channels beyond the last are zero
  for (int i = tid; i < RT * (dp / 4); i += 128) {
    const int quad = i % 4, r = i / 4 % RT, d = i / (4 * RT) * 16 + quad * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows && d < hd)
      x = load4(a.q + ((long long)(t0 + r / a.rep) * a.n_heads + kvh * a.rep + r % a.rep) * hd + d);
    float* dst = qt + d * RT + (RT == 64 ? r ^ quad * 8 : r);
    dst[0] = x.x; dst[RT] = x.y; dst[2 * RT] = x.z; dst[3 * RT] = x.w;
  }
  const int r0 = tid / CG * RPT, c0 = tid % CG * (CPT > 4 ? 4 : CPT);
  int pos[RPT];
  float m[RPT], l[RPT];
#pragma unroll
  for (int i = 0; i < RPT; i++) {
    const int r = r0 + i;
    pos[i] = r < rows ? pos0 + r / a.rep : -1;
    m[i] = -INFINITY;
    l[i] = 0.f;
    if (a.sink && r < rows) {            // the sink as a key of score sink_h whose value is zero
      m[i] = a.sink[kvh * a.rep + r % a.rep];
      l[i] = 1.f;
    }
  }
  float o[VC][RPT][CPT];
#pragma unroll
  for (int v = 0; v < VC; v++)
#pragma unroll
    for (int i = 0; i < RPT; i++)
#pragma unroll
      for (int j = 0; j < CPT; j++) o[v][i][j] = 0.f;

  const int first_win = lo / KT * KT;
  // where the keys of a tile stand in the pools, in rows (-1: no row of the tile sees the key), looked up a tile ahead: the table and
  // the divisions for every piece of a key or value were most of a tile's time
  __shared__ long long row_s[KT];
  auto row_of = [&](int k0) {
    const int j = k0 + tid;
    if (tid >= KT || j > last || !(j >= lo || j < keep)) return -1ll;
    return paged_offset(a.pv, seq, j, kvh) / hd;
  };
  auto after = [&](int k0) { return k0 + KT < first_win && k0 + KT >= keep ? first_win : k0 + KT; };      // from the kept keys on to the window
  int k0 = keep > 0 ? 0 : first_win;
  if (tid < KT) row_s[tid] = row_of(k0);
  __syncthreads();
  for (; k0 <= last;) {
    // values as they are, on their way while the scores are made; keys transposed, eight pieces at a time; keys that no row sees are
    // zero and not read
    for (int i = tid; i < KT * VW / 4; i += 128) {
      const int key = i / (VW / 4), c = i % (VW / 4) * 4;
      const long long row = row_s[key];
      const bool in = c < a.vd && row >= 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(vs + key * VW + c)),
                   "l"(in ? a.v_pool + row * a.v_ld + c : a.v_pool), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int i0 = tid; i0 < KT * (dp / 4); i0 += 8 * 128) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * 128, quad = i % 4, key = i / 4 % KT, d = i / (4 * KT) * 16 + quad * 4;
        x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d < hd && row_s[key] >= 0) x[u] = load4(a.k_pool + row_s[key] * hd + d);
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * 128, quad = i % 4, key = i / 4 % KT, d = i / (4 * KT) * 16 + quad * 4;
        if (d >= dp) break;
        float* dst = kt + d * KT + (key ^ quad * 8);
        dst[0] = x[u].x; dst[KT] = x[u].y; dst[2 * KT] = x[u].z; dst[3 * KT] = x[u].w;
      }
    }
    const int k_next = after(k0);
    const long long row_next = row_of(k_next);
    __syncthreads();
    float s[RPT][CPT];
#pragma unroll
    for (int i = 0; i < RPT; i++)
#pragma unroll
      for (int j = 0; j < CPT; j++) s[i][j] = 0.f;
    for (int d0 = 0; d0 < dp; d0 += 16) {
      float part[RPT][CPT];
#pragma unroll
      for (int d = 0; d < 16; d++) {
        const int turn = d / 4 * 8;
        float x[RPT], y[CPT];
        get(x, qt + (d0 + d) * RT + (RT == 64 ? r0 ^ turn : r0), 0);
        const float* kr = kt + (d0 + d) * KT;
        if constexpr (CPT > 4) {
          float y0[4], y1[4];
          get(y0, kr + (c0 ^ turn), 0);
          get(y1, kr + ((c0 + CSTEP) ^ turn), 0);
#pragma unroll
          for (int j = 0; j < 4; j++) { y[j] = y0[j]; y[CPT - 4 + j] = y1[j]; }
        } else {
          get(y, kr + (c0 ^ turn), 0);
        }
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
          for (int j = 0; j < CPT; j++) part[i][j] = d == 0 ? x[i] * y[j] : fmaf(x[i], y[j], part[i][j]);
      }
#pragma unroll
      for (int i = 0; i < RPT; i++)
#pragma unroll
        for (int j = 0; j < CPT; j++) s[i][j] += part[i][j];
    }
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < CPT; j++) {
        const int key = k0 + c0 + (j & 3) + (j >> 2) * CSTEP;
        float x = s[i][j] * a.scale;
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        s[i][j] = sees(a, pos[i], key) ? x : -INFINITY;
        top = fmaxf(top, s[i][j]);
      }
#pragma unroll
      for (int w = 1; w < CG; w <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
      top = fmaxf(top, m[i]);
      const float fade = m[i] == -INFINITY ? 0.f : expf(m[i] - top);
      // the row's sum in one order for either height of a tile, so that it does not depend on what else is in the step: four
      // neighbouring keys, then the two groups 32 keys apart (a lane's own, or eight lanes apart), then the lanes
      float four[CPT / 4];
#pragma unroll
      for (int j = 0; j < CPT; j++) {
        s[i][j] = s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - top);
        four[j / 4] = j % 4 == 0 ? s[i][j] : four[j / 4] + s[i][j];
      }
      float sum = CPT > 4 ? four[0] + four[CPT / 4 - 1] : four[0] + __shfl_xor_sync(0xffffffffu, four[0], 8);
#pragma unroll
      for (int w = 1; w < 8; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
      l[i] = l[i] * fade + sum;
      m[i] = top;
#pragma unroll
      for (int v = 0; v < VC; v++)
#pragma unroll
        for (int j = 0; j < CPT; j++) o[v][i][j] *= fade;
    }
#pragma unroll
    for (int j = 0; j < CPT; j++) {
      float* dst = pt + (c0 + (j & 3) + (j >> 2) * CSTEP) * RP + r0;
      if constexpr (RPT == 4) *reinterpret_cast<float4*>(dst) = make_float4(s[0][j], s[1][j], s[RPT - 2][j], s[RPT - 1][j]);
      else *reinterpret_cast<float2*>(dst) = make_float2(s[0][j], s[1][j]);
    }
    if (tid < KT) row_s[tid] = row_next;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // keys behind the last one any row sees have weight zero
    const int keys = min(KT, (last - k0 + 16) / 16 * 16);
#pragma unroll
    for (int v = 0; v < VC; v++) {
      for (int j0 = 0; j0 < keys; j0 += 16) {
        float part[RPT][CPT];
#pragma unroll
        for (int key = 0; key < 16; key++) {
          float x[RPT], y[CPT];
          get(x, pt + (j0 + key) * RP + r0, 0);
          get(y, vs + (j0 + key) * VW + v * 64 + c0, CSTEP);
#pragma unroll
          for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < CPT; j++) part[i][j] = key == 0 ? x[i] * y[j] : fmaf(x[i], y[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
          for (int j = 0; j < CPT; j++) o[v][i][j] += part[i][j];
      }
    }
    __syncthreads();
    k0 = k_next;
  }
#pragma unroll
  for (int i = 0; i < RPT; i++) {
    const int r = r0 + i;
    if (r >= rows) continue;
    const int t = t0 + r / a.rep, h = kvh * a.rep + r % a.rep;
    const float inv = 1.0f / l[i];
    float all = 0.f;
#pragma unroll
    for (int v = 0; v < VC; v++)
#pragma unroll
      for (int j = 0; j < CPT; j++) all += o[v][i][j];
    if (!(fabsf(all) < INFINITY)) {
      row_again<VC, CPT, CSTEP>(a, seq, t, h, pos[i], c0, inv);
      continue;
    }
    float* dst = a.out + ((long long)t * a.n_heads + h) * a.vd;
    const float* gate = a.gate ? a.gate + (long long)t * a.gate_ld + (long long)h * a.vd : nullptr;
#pragma unroll
    for (int v = 0; v < VC; v++)
#pragma unroll
      for (int j = 0; j < CPT; j++) {
        const int c = v * 64 + c0 + (j & 3) + (j >> 2) * CSTEP;
        if (c < a.vd) {
          float x = o[v][i][j] * inv;
          if (gate) x *= 1.0f / (1.0f + expf(-gate[c]));
          dst[c] = x;
        }
      }
  }
}

constexpr size_t smem_bytes(int rt, int vc, int hd) {
  const int dp = (hd + 15) / 16 * 16;
  return (size_t)(dp * (rt + KT) + KT * vc * 64 + KT * (rt + 4)) * sizeof(float);
}

template <int RT, int VC>
int launch(const F32Args& a, int n_seqs, int max_q_len, cudaStream_t stream) {
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<RT, VC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem_bytes(RT, VC, 256));
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  const dim3 grid((max_q_len + a.tokens - 1) / a.tokens, a.pv.n_kv_heads, n_seqs);
  attention_f32_kernel<RT, VC><<<grid, 128, smem_bytes(RT, VC, a.pv.head_dim), stream>>>(a);
  return (int)cudaGetLastError();
}
}  // namespace

// Rows in whole 16-byte pieces, key and value rows of up to 256 channels, up to 64 query heads a KV head.
MF_API int mf_attention_f32_ok(int n_heads, int n_kv, int hd, int vd, int v_ld) {
  return n_kv > 0 && n_kv <= 65535 && n_heads % n_kv == 0 && n_heads / n_kv <= 64 && hd > 0 && hd <= 256 && hd % 4 == 0 && vd > 0 &&
         vd <= 256 && vd % 4 == 0 && v_ld % 4 == 0 && v_ld >= vd;
}

// The sequences' rows of q and out start at q_start and are q_len long; row i of the block table is sequence i's; ctx_len
// counts the keys after the step.
MF_API int mf_attention_f32(const float* q, const float* k_pool, const float* v_pool, float* out, const int* q_start,
                            const int* q_len, const int* ctx_len, int n_seqs, int max_q_len, int n_heads, int n_kv, int hd,
                            const int* block_table, int bt_stride, int page_size, float scale, int window, int vd, int v_ld,
                            int keep_first, const float* sink, const float* gate, long long gate_ld, float softcap,
                            cudaStream_t stream) {
  if (n_seqs <= 0 || max_q_len <= 0) return 0;
  if (!mf_attention_f32_ok(n_heads, n_kv, hd, vd, v_ld) || n_seqs > 65535 || keep_first < 0 || (((uintptr_t)q) & 15) ||
      (((uintptr_t)k_pool) & 15) || (((uintptr_t)v_pool) & 15))
    return MF_ERR_BAD_ARG;
  mf_count(MF_K_ATTN_GENERIC);
  mf_count(MF_K_ATTN_F32);
  const int rep = n_heads / n_kv, vc = (vd + 63) / 64;
  // The tallest tile that leaves an SM a block and a half: a block is a warp a scheduler, which waits for itself; 16 rows where they hold
  // all there is, as in decoding.  Heads of 128, 150 tokens behind 300 keys: 32 / 8 heads 202 us in 80 blocks of 64 rows, 102 in 152 of 32,
  // 104 in 304 of 16; 16 / 4 heads 212 in 40, 99 in 76, 75 in 152.
  const int sms = mf_sm_count();
  auto crowded = [&](int rows) {
    return rep <= rows && (long long)((max_q_len + rows / rep - 1) / (rows / rep)) * n_kv * n_seqs * 2 > 3ll * sms;
  };
  const int height = (long long)max_q_len * rep <= 16 ? 16 : crowded(64) ? 64 : crowded(32) ? 32 : rep <= 16 ? 16 : rep <= 32 ? 32 : 64;
  F32Args a{q, k_pool, v_pool, out, q_start, q_len, ctx_len, PagedView{block_table, bt_stride, page_size, n_kv, hd},
            n_heads, rep, height / rep, scale, window, vd, v_ld, keep_first, sink, gate, gate_ld, softcap};
#define F32_GO(RT)                                              \
  do {                                                          \
    if (vc == 1) return launch<RT, 1>(a, n_seqs, max_q_len, stream); \
    if (vc == 2) return launch<RT, 2>(a, n_seqs, max_q_len, stream); \
    if (vc == 3) return launch<RT, 3>(a, n_seqs, max_q_len, stream); \
    return launch<RT, 4>(a, n_seqs, max_q_len, stream);         \
  } while (0)
  if (height == 16) F32_GO(16);
  if (height == 32) F32_GO(32);
  F32_GO(64);
#undef F32_GO
}
