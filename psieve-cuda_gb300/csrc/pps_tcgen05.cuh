// pps_tcgen05.cuh -- the fifth-generation tensor core instructions the tensor
// walk uses (sm_103a inline PTX): TMEM allocation, one-CTA fp16 MMA with f32
// accumulators, commit to an mbarrier, TMEM loads, and the mbarrier itself.
#pragma once
#include <stdint.h>

namespace pps {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// One attempt: the hardware suspends the thread for a limited time.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0u;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar, uint32_t count = 1u) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// The same by lane 0 of a warp (a predicate, not a branch).
__device__ __forceinline__ void mbar_arrive_lane0(uint32_t bar, uint32_t count = 1u) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.u32 p, %2, 0;\n\t"
      "@p mbarrier.arrive.release.cta.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
      "r"(count), "r"(threadIdx.x & 31u)
      : "memory");
}
// Waits for a phase of the barrier, with a limit: false when the bound's clocks
// ran out or another role that shares it gave up (give_up != 0, set here on a
// time-out), so that every role then leaves its loops and the kernel ends.  The
// votes keep the branches uniform.  PAUSE: ns to sleep between attempts, for the
// roles that run ahead, so that their polling takes no issue slots from the
// others.
struct MbarBound {  // in shared memory
  long long limit;
  uint32_t give_up;
};
template <uint32_t PAUSE>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile MbarBound* bound) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
#pragma unroll 1
  for (uint32_t i = 1;; ++i) {
    if (PAUSE) __nanosleep(PAUSE);
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 0u) {
      if (clock64() - t0 > bound->limit) bound->give_up = 1u;
      if (__any_sync(0xffffffffu, bound->give_up != 0u)) return false;
    }
  }
}

// ---- TMEM
// One whole warp; ncols a power of two from 32; the address goes to shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 64 (48) columns of this warp's 32 TMEM lanes, the low 16 bits of each value, two
// columns to a register (column 2i in the low half of r[i]); waits for them.
__device__ __forceinline__ void tmem_ld64_lo16(uint32_t* r, uint32_t tmem) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.pack::16b.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]), "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23]), "=&r"(r[24]), "=&r"(r[25]), "=&r"(r[26]), "=&r"(r[27]), "=&r"(r[28]), "=&r"(r[29]), "=&r"(r[30]), "=&r"(r[31])
      : "r"(tmem)
      : "memory");
}
__device__ __forceinline__ void tmem_ld48_lo16(uint32_t* r, uint32_t tmem) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%25];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]), "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23])
      : "r"(tmem), "r"(tmem + 32u)
      : "memory");
}
// 16 columns of this warp's 32 TMEM lanes from registers.
__device__ __forceinline__ void tmem_st16(uint32_t tmem, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(tmem),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- MMA: D[128 x n] (f32, TMEM) (+)= A[128 x 16] B[n x 16]^T, fp16.  A lies
// in TMEM: lane = row, two K elements to a column (8 columns).  B is K-major in
// shared memory without swizzle: 8 x 16-byte core matrices of 128 contiguous
// bytes, `sbo` bytes between 8-row groups, `lbo` bytes between the two
// 8-element halves of K.
// The descriptor's words: lo (address and lbo), hi (sbo, descriptor version 1).
__device__ __forceinline__ uint32_t mma_desc_lo(uint32_t addr, uint32_t lbo) {
  return ((addr >> 4) & 0x3fffu) | (((lbo >> 4) & 0x3fffu) << 16);
}
__device__ __forceinline__ uint32_t mma_desc_hi(uint32_t sbo) { return ((sbo >> 4) & 0x3fffu) | (1u << 14); }
// D f32, A and B f16, M 128; neg: the product with -A
__device__ __forceinline__ uint32_t mma_idesc_f16(uint32_t n, bool neg) {
  return (1u << 4) | ((uint32_t)neg << 13) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// D = A_l B, then D += A_h B (`a_tmem` is A_l's column, A_h's is 8 further); the
// mbarrier arrives when both are done, and every MMA issued before.  The whole
// warp, one lane issues.
__device__ __forceinline__ void mma_pair_f16(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi,
                                             uint32_t idesc_l, uint32_t idesc_h, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e, f, t;\n\t.reg .b64 b;\n\t"
      "mov.b64 b, {%3, %4};\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 f, 0, 0;\n\t"
      "setp.eq.b32 t, 0, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %5, f;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], b, %6, t;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%7];\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(a_tmem + 8u), "r"(b_lo), "r"(b_hi), "r"(idesc_l), "r"(idesc_h), "r"(bar)
      : "memory");
}
// The mbarrier arrives when every MMA issued before is done (the same lane).
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}

}  // namespace pps
