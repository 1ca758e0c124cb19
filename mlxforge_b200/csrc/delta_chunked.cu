// The gated delta rule over runs of tokens (see delta_rule.cu for the rule itself).
//
// Per head, with the decays g_t of a run of R tokens, their running products G_t = g_1 .. g_t (per key channel) and
// the state S_0 before the run, the rule unrolls to
//
//   U = T V - W S_0 ,   O = Qh S_0 + B U ,   S_R = G_R S_0 + Kt^T U
//
//   A[t][s] = sum_c k_t k_s (G_t / G_s) (s < t) ,   B[t][s] = sum_c q_t k_s (G_t / G_s) (s <= t) ,
//   T = (1 + diag(beta) A)^-1 diag(beta) ,  W = T (G k) ,  Qh = G q ,  Kt_s = k_s G_R / G_s .
//
// Everything but the three products with the state is independent of it, so it is made for all runs side by side
// (delta_runs_kernel), and only those products go from run to run (delta_state_kernel).  Every quotient of decays is
// formed as the product of the decays between the two tokens, never by dividing, so nothing overflows however
// strong the decays are.  All of it is IEEE 32-bit.
//
// Why: the recurrence token after token is bound by one token's chain of instructions (0.30 us a token, the FMA pipe 8 %
// busy at heads of 128); a run of 16 tokens makes of it three small matrix products.  2,048 tokens of 16 heads of
// 128 x 128: 615 -> 192 us (48 + 144); 8 heads: 613 -> 132 us (25 + 107).  What bounds it now is shared memory, which hands
// every lane four bytes a cycle at most, broadcast or not: 1,540 of the 2,200 cycles of a run are its loads (tiles of 4 x 4
// results read eight numbers for sixteen multiplications; counters: its pipe 68 % busy, the FMA pipe 42 %).
#include "common.cuh"

namespace {
constexpr int R = 16;                  // tokens of a run
constexpr int STAGES = 4;              // runs whose operands are in shared memory or on their way
constexpr int WAIT_LIMIT = 1 << 22;    // polls of a barrier before a thread gives up

// floats that a run of one head hands from the first kernel to the second: W [D][16], Qh [D][16], Kt [16][D], G_R [D],
// B [16][16], then T V [vdim / NC][16][NC].  The channels of Kt and G_R stand in the order of place().
constexpr int common_floats(int D) { return D * 2 * R + R * D + D + R * R; }
// Where channel d of a row of Kt and G_R stands: the channels d, d + P, d + 2P, .. (P = 8) that a thread of the second
// kernel owns are neighbours.  DT of them at D channels.
template <int D>
__device__ __forceinline__ int place(int d) {
  constexpr int DT = D / 32;
  return d / (8 * DT) * (8 * DT) + (d % 8) * DT + d / 8 % DT;
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, int* status) {
  for (int i = 0; i < WAIT_LIMIT; i++) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  if (status) atomicExch(status, 61);
  return false;
}

// keeps the loads of an unrolled loop's turns from being gathered in front of it (registers)
__device__ __forceinline__ void turn_ends() { asm volatile("" ::: "memory"); }

// N neighbouring floats (2 or 4, aligned to their size) between registers and shared memory in one access
template <int N>
__device__ __forceinline__ void get(float (&x)[N], const float* p) {
  if constexpr (N == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
  } else if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    x[0] = t.x; x[1] = t.y;
  } else {
    x[0] = *p;
  }
}
template <int N>
__device__ __forceinline__ void put(float* p, const float (&x)[N]) {
  if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  else if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  else *p = x[0];
}

// the sequence that owns run `i` of the launch, and the run's index within it; false behind the last run
__device__ __forceinline__ bool find_run(int i, const int* __restrict__ q_len, int n_seqs, int& seq, int& run) {
  for (seq = 0; seq < n_seqs; seq++) {
    const int runs = (q_len[seq] + R - 1) / R;
    if (i < runs) {
      run = i;
      return true;
    }
    i -= runs;
  }
  return false;
}

// ---------------------------------------------------------------------------- what does not depend on the state
// A block of D threads per (run, head).  A thread loads a channel of all tokens; for A and B a warp walks some of the
// tokens s forward through the run at once, p_s = k_s times the decays since, D/32 channels a lane, and sums over its lanes
// token by token, so that a row read from shared memory serves all of its s and nothing is accumulated in registers.
template <int D>
__global__ void __launch_bounds__(D, 1024 / D)
delta_runs_kernel(const float* __restrict__ qkv, const float* __restrict__ beta, const float* __restrict__ ag, int ag_ld,
                  const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, int n_seqs,
                  float* __restrict__ runs_out, int n_heads, int n_kv, int vdim, int nc) {
  constexpr int WARPS = D / 32, CH = D / 32, SP = R / WARPS;       // channels of a lane; tokens s of a warp
  __shared__ __align__(16) float kqs[2][R][D], gs[R][D];
  __shared__ __align__(16) float AB[2][R][R], Tm[R][R];
  __shared__ float bs[R];
  float(*ks)[D] = kqs[0];
  float(*qs)[D] = kqs[1];
  const int h = blockIdx.y, c = threadIdx.x, warp = c >> 5, lane = c & 31;
  int seq, run;
  if (!find_run(blockIdx.x, seq_q_len, n_seqs, seq, run)) return;
  const int kvh = h / (n_heads / n_kv);
  const int C = 2 * n_kv * D + n_heads * vdim;
  const long long t0 = seq_q_start[seq] + run * R;
  const int nt = min(R, seq_q_len[seq] - run * R);
  float* out = runs_out + ((long long)blockIdx.x * n_heads + h) * (common_floats(D) + R * vdim);
  float* out_kt = out + D * 2 * R;
  float* out_g = out_kt + R * D;
  float* out_b = out_g + D;
  float* out_tv = out_b + R * R;
  if (c < R) bs[c] = c < nt ? beta[(t0 + c) * n_heads + h] : 0.f;
  {
    const float* row = qkv + t0 * C + kvh * D + c;
    const float* grow = ag + t0 * ag_ld + h * D + c;
#pragma unroll
    for (int t = 0; t < R; t++) {
      const bool in = t < nt;
      qs[t][c] = in ? row[(long long)t * C] : 0.f;
      ks[t][c] = in ? row[(long long)t * C + n_kv * D] : 0.f;
      gs[t][c] = in ? grow[(long long)t * ag_ld] : 1.f;
    }
  }
  __syncthreads();
  {
    float p[SP][CH];
#pragma unroll
    for (int j = 0; j < SP; j++)
#pragma unroll
      for (int i = 0; i < CH; i++) p[j][i] = 0.f;
#pragma unroll 2
    for (int t = 0; t < R; t++) {
      float k[CH], q[CH], g[CH];
      get(k, &ks[t][lane * CH]);
      get(q, &qs[t][lane * CH]);
      get(g, &gs[t][lane * CH]);
      float x[2 * SP];                     // A[t][s] of the warp's s = warp + WARPS j, then B[t][s]
#pragma unroll
      for (int j = 0; j < SP; j++) {
        const bool own = t == warp + WARPS * j;
#pragma unroll
        for (int i = 0; i < CH; i++) p[j][i] = own ? k[i] : p[j][i] * g[i];
        x[j] = k[0] * p[j][0];
        x[SP + j] = q[0] * p[j][0];
#pragma unroll
        for (int i = 1; i < CH; i++) {
          x[j] = fmaf(k[i], p[j][i], x[j]);
          x[SP + j] = fmaf(q[i], p[j][i], x[SP + j]);
        }
      }
      // sums over the lanes: each step a lane keeps half of its values and hands the other half on
      int m = 16, idx = 0;
#pragma unroll
      for (int n = SP; n >= 1; n >>= 1, m >>= 1) {
        const bool up = lane & m;
        idx = 2 * idx + (up ? 1 : 0);
#pragma unroll
        for (int i = 0; i < n; i++) {
          const float keep = up ? x[n + i] : x[i], give = up ? x[i] : x[n + i];
          x[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
      }
      for (; m >= 1; m >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], m);
      if ((lane & (16 / SP - 1)) == 0) AB[idx / SP][t][warp + WARPS * (idx % SP)] = x[0];
    }
  }
  __syncthreads();
  if (c < R) {
    // column c of T: (1 + diag(beta) A) x = beta_c e_c, from the top down
    float x[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
      float d0 = 0.f, d1 = 0.f;
#pragma unroll
      for (int s = 0; s < i; s++) {
        if (s & 1) d1 = fmaf(AB[0][i][s], x[s], d1);
        else d0 = fmaf(AB[0][i][s], x[s], d0);
      }
      x[i] = i < c ? 0.f : (i == c ? bs[i] : 0.f) - bs[i] * (d0 + d1);
      if (i % 4 == 3) turn_ends();
    }
#pragma unroll
    for (int i = 0; i < R; i++) Tm[i][c] = x[i];
  } else {
    // meanwhile the rest writes what is done: B (what stands at s > t is not read)
    for (int i = c - R; i < R * R; i += D - R) out_b[i] = AB[1][i / R][i % R];
  }
  float kh[R], w[R], qh[R];
  {
    float G = 1.f;
#pragma unroll
    for (int t = 0; t < R; t++) {
      const float k = ks[t][c], g = gs[t][c];
      w[t] = k;
      G *= g;
      kh[t] = G * k;
      qh[t] = G * qs[t][c];
    }
    float after = 1.f;                     // product of the decays behind a token
#pragma unroll
    for (int t = R - 1; t >= 0; t--) {
      out_kt[t * D + place<D>(c)] = w[t] * after;
      after *= gs[t][c];
    }
    out_g[place<D>(c)] = after;
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < R; t++) {
    float acc = 0.f;
#pragma unroll
    for (int s = 0; s <= t; s++) acc = fmaf(Tm[t][s], kh[s], acc);
    w[t] = acc;
    if (t % 4 == 3) turn_ends();
  }
  {
    // a thread has a row of 16 of W and of Qh: through shared memory (16-byte pieces of neighbouring rows in turned
    // places), so that a warp writes whole lines
    float4* stage = reinterpret_cast<float4*>(&kqs[0][0][0]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      stage[c * 4 + (j ^ (c >> 1 & 3))] = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
      stage[(D + c) * 4 + (j ^ (c >> 1 & 3))] = make_float4(qh[4 * j], qh[4 * j + 1], qh[4 * j + 2], qh[4 * j + 3]);
    }
    __syncthreads();
    float4* dst = reinterpret_cast<float4*>(out);
#pragma unroll
    for (int i = c; i < 8 * D; i += D) {
      const int row = i / 4;
      dst[i] = stage[row * 4 + ((i & 3) ^ (row >> 1 & 3))];
    }
  }
  for (int col = c; col < vdim; col += D) {
    float v[R];
    const float* row = qkv + t0 * C + 2 * n_kv * D + h * vdim + col;
#pragma unroll
    for (int t = 0; t < R; t++) v[t] = t < nt ? row[(long long)t * C] : 0.f;
    float* dst = out_tv + (col / nc) * R * nc + col % nc;
#pragma unroll
    for (int t = 0; t < R; t++) {
      float acc = 0.f;
#pragma unroll
      for (int s = 0; s <= t; s++) acc = fmaf(Tm[t][s], v[s], acc);
      dst[t * nc] = acc;
      if (t % 4 == 3) turn_ends();
    }
  }
}

// ---------------------------------------------------------------------------- from run to run
// A block owns NC columns of a head's state.  Its first four warps go from run to run with U = T V - W S and
// S = G S + Kt^T U, a thread D/32 x NC/4 of S in registers and once more in shared memory for the next product; the other
// four follow one run behind with O = Qh S + B U, so that nothing of the read-out is in the chain from run to run.  In
// both products over the channels a half-warp takes every eighth channel and a thread 4 x NC/4 results, and the eight
// partial sums meet in shared memory.  Operands arrive as two bulk copies a run into a ring of four stages.
template <int D, int NC>
__global__ void __launch_bounds__(256, 1)
delta_state_kernel(const float* __restrict__ runs, float* __restrict__ state, long long state_stride,
                   const int* __restrict__ seq_q_start, const int* __restrict__ seq_q_len, const int* __restrict__ slots,
                   float* __restrict__ o_out, int n_heads, int vdim, int* __restrict__ status) {
  constexpr int COMMON = common_floats(D), STAGE = COMMON + R * NC;
  constexpr int CT = NC / 4;               // columns of a thread's tile
  constexpr int DT = D / 32;               // channels of a thread's tile of the state
  constexpr int RS = NC + 4;               // a row of partial sums, padded: no two rows of a store in the same banks
  extern __shared__ __align__(128) float sm[];
  float* S_s = sm + STAGES * STAGE;        // [3][D][NC]
  float* U_s = S_s + 3 * D * NC;           // [2][16][NC]
  float* red = U_s + 2 * R * NC;           // [2][8][16][RS]
  __shared__ __align__(8) unsigned long long bars[STAGES];
  const int seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * NC;
  const bool reads = threadIdx.x >= 128;   // one of the read-out's warps
  const int tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31;
  const int n = seq_q_len[seq];
  const int n_runs = (n + R - 1) / R;
  long long first = 0;
  for (int i = 0; i < seq; i++) first += (seq_q_len[i] + R - 1) / R;
  const long long run_floats = COMMON + (long long)R * vdim;
  const float* src = runs + (first * n_heads + h) * run_floats;
  const unsigned bar0 = smem_u32(bars);
  const bool fetches = threadIdx.x == 128;
  if (fetches) {
    for (int s = 0; s < STAGES; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar0 + 8 * s));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  auto fetch = [&](int run) {
    const unsigned bar = bar0 + 8 * (run % STAGES), dst = smem_u32(sm + (run % STAGES) * STAGE);
    const float* from = src + (long long)run * n_heads * run_floats;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((unsigned)(STAGE * 4)) : "memory");
    bulk_copy(dst, from, COMMON * 4, bar);
    bulk_copy(dst + COMMON * 4, from + COMMON + (long long)blockIdx.z * R * NC, R * NC * 4, bar);
  };
  if (fetches)
    for (int r = 0; r < 2 && r < n_runs; r++) fetch(r);
  // the thread's tile of the state: channels d0, d0 + 8, ..; columns c0 .. c0 + CT
  const int d0 = warp * 8 * DT + (lane >> 2), c0 = (lane & 3) * CT;
  float* S = state + (long long)slots[seq] * state_stride + (long long)h * D * vdim + col0 + c0;
  float st[DT][CT];
  if (!reads) {
#pragma unroll
    for (int i = 0; i < DT; i++) {
#pragma unroll
      for (int j = 0; j < CT; j++) st[i][j] = S[(long long)(d0 + 8 * i) * vdim + j];
      put(S_s + (d0 + 8 * i) * NC + c0, st[i]);
    }
  }
  float* o = o_out + (long long)seq_q_start[seq] * n_heads * vdim + h * vdim + col0;
  constexpr int PER = R * NC / 128;        // results of a thread where partial sums meet
  const int pr = tid * PER / NC, pc = tid * PER % NC;
  float* my_red = red + (reads ? 8 * R * RS : 0);
  const int half = lane >> 4, r0 = (lane >> 2 & 3) * 4;
  // rows r0 .. r0 + 4 of M [16][D] (as [D][16]) times S, the channels 8 i + 2 warp + half; the partial sums to my_red
  auto product = [&](const float* m, const float* s) {
    m += (2 * warp + half) * R + r0;
    s += (2 * warp + half) * NC + c0;
    float acc[4][CT];
#pragma unroll
    for (int k0 = 0; k0 < D / 8; k0 += 8) {
      // chains of eight channels, then their sums: as short as the ones of the recurrence token after token
      float part[4][CT];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        float a[4], b[CT];
        get(a, m + (k0 + k) * 8 * R);
        get(b, s + (k0 + k) * 8 * NC);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < CT; j++) part[i][j] = k == 0 ? a[i] * b[j] : fmaf(a[i], b[j], part[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < CT; j++) acc[i][j] = k0 == 0 ? part[i][j] : acc[i][j] + part[i][j];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) put(my_red + ((2 * warp + half) * R + r0 + i) * RS + c0, acc[i]);
  };
  auto meet = [&](float (&x)[PER]) {       // the eight partial sums of the thread's results, in their order
    float part[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) x[j] = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      get(part, my_red + (w * R + pr) * RS + pc);
#pragma unroll
      for (int j = 0; j < PER; j++) x[j] += part[j];
    }
  };
  __syncthreads();
  for (int i = 0; i <= n_runs; i++) {
    if (!reads) {
      if (i < n_runs) {
        const float* op = sm + (i % STAGES) * STAGE;
        float* u_s = U_s + (i & 1) * R * NC;
        bar_wait(bar0 + 8 * (i % STAGES), (i / STAGES) & 1, status);
        product(op, S_s + (i % 3) * D * NC);
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        float ws[PER], u[PER];
        meet(ws);
        get(u, op + COMMON + pr * NC + pc);
#pragma unroll
        for (int j = 0; j < PER; j++) u[j] -= ws[j];
        put(u_s + pr * NC + pc, u);
        const float* kt = op + D * 2 * R + (warp * 8 + (lane >> 2)) * DT;
        float g[DT];
        get(g, kt + R * D);
#pragma unroll
        for (int a = 0; a < DT; a++)
#pragma unroll
          for (int j = 0; j < CT; j++) st[a][j] *= g[a];
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
        for (int t = 0; t < R; t++) {
          float k[DT], ut[CT];
          get(k, kt + t * D);
          get(ut, u_s + t * NC + c0);
#pragma unroll
          for (int a = 0; a < DT; a++)
#pragma unroll
            for (int j = 0; j < CT; j++) st[a][j] = fmaf(k[a], ut[j], st[a][j]);
        }
        float* next = S_s + ((i + 1) % 3) * D * NC;
#pragma unroll
        for (int a = 0; a < DT; a++) put(next + (d0 + 8 * a) * NC + c0, st[a]);
      }
    } else {
      // stage i + 2 was read last one turn ago, by these warps, and the barrier at the turn's end lies between
      if (fetches && i + 2 < n_runs) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        fetch(i + 2);
      }
      if (i > 0) {
        const int run = i - 1;
        const float* op = sm + (run % STAGES) * STAGE;
        const float* u_s = U_s + (run & 1) * R * NC;
        bar_wait(bar0 + 8 * (run % STAGES), (run / STAGES) & 1, status);
        product(op + D * R, S_s + (run % 3) * D * NC);
        // B U while the partial sums are on their way, each row over its own tokens and the ones before: a zero of B would let
        // what is not finite of a later token into it
        float x[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) x[j] = 0.f;
        const float* bm = op + D * 2 * R + R * D + D + pr * R;
#pragma unroll
        for (int s = 0; s < R; s += 4) {
          float b[4], u[PER];
          get(b, bm + s);
#pragma unroll
          for (int k = 0; k < 4; k++) {
            get(u, u_s + (s + k) * NC + pc);
#pragma unroll
            for (int j = 0; j < PER; j++)
              if (s + k <= pr) x[j] = fmaf(b[k], u[j], x[j]);
          }
        }
        asm volatile("bar.sync 2, 128;\n" ::: "memory");
        float qs[PER];
        meet(qs);
        if (run * R + pr < n) {
#pragma unroll
          for (int j = 0; j < PER; j++) x[j] += qs[j];
          put(o + (long long)(run * R + pr) * n_heads * vdim + pc, x);
        }
      }
    }
    __syncthreads();
  }
  if (!reads) {
#pragma unroll
    for (int i = 0; i < DT; i++)
#pragma unroll
      for (int j = 0; j < CT; j++) S[(long long)(d0 + 8 * i) * vdim + j] = st[i][j];
  }
}

template <int D, int NC>
int launch_state(const float* runs, float* state, long long state_stride, const int* seq_q_start, const int* seq_q_len,
                 const int* slots, float* o_out, int n_seqs, int n_heads, int vdim, int* status, cudaStream_t stream) {
  constexpr size_t smem =
      (size_t)(STAGES * (common_floats(D) + R * NC) + 3 * D * NC + 2 * R * NC + 2 * 8 * R * (NC + 4)) * sizeof(float);
  static DeviceOnce once;
  const int dev = mf_current_device();
  if (dev < 0) return MF_ERR_BAD_ARG;
  if (!once.done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(delta_state_kernel<D, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    once.done[dev] = true;
  }
  delta_state_kernel<D, NC><<<dim3(n_seqs, n_heads, vdim / NC), 256, smem, stream>>>(
      runs, state, state_stride, seq_q_start, seq_q_len, slots, o_out, n_heads, vdim, status);
  return (int)cudaGetLastError();
}
}  // namespace

// Heads of 64 or 128 channels whose values are whole blocks of 16 columns.
MF_API int mf_delta_runs_ok(int dim, int vdim) { return (dim == 64 || dim == 128) && vdim > 0 && vdim % 16 == 0; }

// Floats of scratch for portions that make `n_runs` runs of 16 tokens in all (every portion's last run may be short).
MF_API long long mf_delta_runs_scratch(long long n_runs, int n_heads, int dim, int vdim) {
  return n_runs * n_heads * (common_floats(dim) + (long long)R * vdim);
}

// qkv, beta, ag, state, o_out as for mf_delta_recurrence.  `n_runs`: the sum of ceil(q_len / 16) over the sequences.
MF_API int mf_delta_recurrence_runs(const float* qkv, const float* beta, const float* ag, int ag_ld, float* state,
                                    long long state_stride, const int* seq_q_start, const int* seq_q_len,
                                    const int* slots, float* o_out, int n_seqs, int n_runs, int n_heads, int n_kv, int dim,
                                    int vdim, float* scratch, int* status, cudaStream_t stream) {
  if (n_seqs <= 0 || n_runs <= 0) return 0;
  if (!mf_delta_runs_ok(dim, vdim) || n_kv <= 0 || n_heads % n_kv || n_heads > 65535 || ((uintptr_t)scratch & 15))
    return MF_ERR_BAD_ARG;
  mf_count(MF_K_DELTA_RECURRENCE);
  mf_count(MF_K_DELTA_RUNS);
  // blocks of 8 columns where blocks of 16 would leave half of the SMs without one (a run takes 0.83 us instead of
  // 1.12 us, so two blocks of 8 after one another are slower than one of 16)
  const int nc = (long long)n_seqs * n_heads * (vdim / 16) * 2 <= mf_sm_count() ? 8 : 16;
#define RUNS_GO(D)                                                                                                    \
  do {                                                                                                                \
    delta_runs_kernel<D><<<dim3(n_runs, n_heads), D, 0, stream>>>(qkv, beta, ag, ag_ld, seq_q_start, seq_q_len, n_seqs, \
                                                                  scratch, n_heads, n_kv, vdim, nc);                  \
    cudaError_t e = cudaGetLastError();                                                                               \
    if (e != cudaSuccess) return (int)e;                                                                              \
    if (nc == 8)                                                                                                      \
      return launch_state<D, 8>(scratch, state, state_stride, seq_q_start, seq_q_len, slots, o_out, n_seqs, n_heads,  \
                                vdim, status, stream);                                                                \
    return launch_state<D, 16>(scratch, state, state_stride, seq_q_start, seq_q_len, slots, o_out, n_seqs, n_heads,   \
                               vdim, status, stream);                                                                 \
  } while (0)
  if (dim == 64) RUNS_GO(64);
  RUNS_GO(128);
#undef RUNS_GO
}
