// The 5th-generation tensor core and bulk-copy primitives the exact integer GEMMs
// (the FirstDim scan, the cascade's key switches) are written with: bounded
// mbarrier waits, bulk copies into shared memory, tcgen05.mma kind::i8 and the
// TMEM loads of their epilogues.
#pragma once
#include "common.cuh"

namespace via {

constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s per wait
constexpr unsigned WAIT_SPINS = 1u << 26;

__device__ __forceinline__ u32 smem_addr(const void* p) { return (u32)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(u64* bar, u32 count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(u64* bar, u32 bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(u64* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(u64* bar, u32 parity) {
  u32 ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase of `parity` to complete. Gives up (false) after WAIT_NS,
// after WAIT_SPINS polls, or, when `honor_abort`, once another role of the CTA
// has aborted.
static __device__ bool mbar_wait(u64* bar, u32 parity, volatile int* abort_flag, bool honor_abort = true) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 1; it < WAIT_SPINS; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 31) == 0) {
      if (honor_abort && *abort_flag) return false;
      if (global_ns() - t0 > WAIT_NS) return false;
    }
  }
  return false;
}

// The test hook's wait: polls a barrier that no thread or copy ever completes
// until `limit_ns` has passed (or WAIT_SPINS polls), then reports failure.
static __device__ bool mbar_wait_never(u64* bar, unsigned limit_ns) {
  const unsigned long long t0 = global_ns();
  for (unsigned it = 0; it < WAIT_SPINS; ++it) {
    if (mbar_try_wait(bar, 0)) return true;
    if ((it & 31) == 0 && global_ns() - t0 > limit_ns) return false;
  }
  return false;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, u32 bytes, u64* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, K-major without swizzle: 8-row x 16-byte
// core matrices, `lbo` bytes between the two core matrices of a 32-byte K
// slice, `sbo` bytes between 8-row groups.
__device__ __forceinline__ u64 smem_desc(u32 addr, u32 lbo, u32 sbo) {
  return (u64)((addr >> 4) & 0x3FFF) | ((u64)((lbo >> 4) & 0x3FFF) << 16) | ((u64)((sbo >> 4) & 0x3FFF) << 32) |
         (1ull << 46);
}

// kind::i8 instruction descriptor: unsigned A and B, K-major, S32 accumulator, M = 128.
__device__ __forceinline__ u32 idesc_u8(int n) { return (2u << 4) | ((u32)(n >> 3) << 17) | ((u32)(128 >> 4) << 24); }

__device__ __forceinline__ void mma_i8(u32 d_tmem, u64 adesc, u64 bdesc, u32 idesc, u32 accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(u64* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld4(u32 taddr, u32 (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(u32 taddr, u32 (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(u32 taddr, u32 (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
template <int W>
__device__ __forceinline__ void tmem_ld(u32 taddr, u32 (&r)[W]) {
  if constexpr (W == 4)
    tmem_ld4(taddr, r);
  else
    tmem_ld8(taddr, r);
}
// Orders later uses of r after the wait above (the loads' results are only
// defined once tcgen05.wait::ld has returned).
template <int K>
__device__ __forceinline__ void pin(u32 (&r)[K]) {
#pragma unroll
  for (int x = 0; x < K; ++x) asm volatile("" : "+r"(r[x]));
}

}  // namespace via
