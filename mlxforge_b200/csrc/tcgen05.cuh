// What attention_talking_prompt.cu and gemm_tcgen05.cu share of the 5th-generation tensor cores: barriers in shared memory, tensor copies,
// descriptors of operands in shared memory, products sent by an elected lane; and how the former waits (with a limit) and reads results
// back.  The other kernels on these units keep helpers of their own: they send from one lane, where an elected one gained nothing or cost time.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace tc5 {

// A turn of a wait lets the warp sleep for up to WAIT_NS: without the hint a turn is short, and warps that wait for each other's products take
// every other issue slot of the ones that work.  WAIT_LIMIT turns are a second or two.
constexpr unsigned WAIT_LIMIT = 1u << 16, WAIT_NS = 20000;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, int code) {
  for (unsigned i = 0; i < WAIT_LIMIT; i++) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity), "r"(WAIT_NS) : "memory");
    if (done) return true;
  }
  if (status) atomicExch(status, code);
  return false;
}
// a look without a wait, so that its answer is on its way while products are sent
__device__ __forceinline__ bool mbar_peek(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void fence_proxy() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// An operand in shared memory in lines of 128 bytes with the 128-byte swizzle, eight lines (1024 bytes) to a group.  K-major: a line is
// 64 values along the contraction, lines are rows.  M- or N-major: a line is 64 values along M or N, lines are the contraction's indices;
// the next 64 values along M or N stand `span_bytes` further.
__device__ __forceinline__ unsigned long long smem_desc(uint32_t addr, uint32_t span_bytes = 16) {
  unsigned long long d = 0;
  d |= (unsigned long long)((addr >> 4) & 0x3FFF);
  d |= (unsigned long long)(span_bytes >> 4) << 16;
  d |= (unsigned long long)(1024 >> 4) << 32;                // eight lines
  d |= (unsigned long long)1 << 46;                          // descriptor version of this architecture
  d |= (unsigned long long)2 << 61;                          // 128-byte swizzle
  return d;
}
// 32-bit sums of bfloat16 products, M x N; A or B along M or N instead of K
__host__ __device__ constexpr uint32_t bf16_idesc(int m, int n, bool a_along_m = false, bool b_along_n = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (a_along_m ? 1u << 15 : 0u) | (b_along_n ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
// Products, their commits and copies are sent by ONE lane, but called by the whole warp with the same operands: the hardware takes them from
// the warp's uniform registers.  Inside `if (lane == 0)` each operand is first moved there from the lane's own, 68 cycles a product of N 64
// instead of 51, and 158 instead of 56 where other warps keep the scheduler busy with multiply-adds.
__device__ __forceinline__ void umma(uint32_t tmem_c, unsigned long long da, unsigned long long db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_c), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile(
      "{\n.reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void expect_tx_one(uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n.reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_3d_one(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "{\n.reg .pred e;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n}\n"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// a value that all lanes have, known to the compiler as such
template <typename T>
__device__ __forceinline__ T uniform(T x) { return __shfl_sync(0xffffffffu, x, 0); }
// by one warp; the columns' base lands in `slot`
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(cols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// 16 columns of the warp's 32 lanes, a lane a thread; the load is on its way until tmem_landed
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
        "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]),
        "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}
// waits for every load of the warp; names the registers, so that no use of them moves above it
template <int N>
__device__ __forceinline__ void tmem_landed(uint32_t (&u)[N]) {
  static_assert(N % 8 == 0, "by eights");
  tmem_wait_ld();
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+r"(u[i]), "+r"(u[i + 1]), "+r"(u[i + 2]), "+r"(u[i + 3]), "+r"(u[i + 4]), "+r"(u[i + 5]), "+r"(u[i + 6]), "+r"(u[i + 7]));
}
// 16 lanes x 16 columns: a thread has lane / 4 and lane / 4 + 8 of the 16 lanes, two neighbouring columns 2 (lane % 4) of either eight:
// u[4 e + 2 r + c] is column 8 e + 2 (lane % 4) + c of lane / 4 + 8 r
__device__ __forceinline__ void tmem_ld_16x16_issue(uint32_t taddr, uint32_t (&u)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
               : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_less() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N)); }

}  // namespace tc5
