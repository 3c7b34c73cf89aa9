// staging.cuh -- mbarriers and bulk copies of the sweeps that stage their operands through shared
// memory (solver_kernels.cu, trsv_local.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#define VSHE_E_TIMEOUT_DEV (-10)

namespace vshe {

// polls of a bounded device-side wait: bar[2..3] of the batch's barrier words
__device__ __forceinline__ unsigned long long spin_limit_of(const unsigned *bar) {
  return *((const volatile unsigned long long *)(bar + 2));
}

// mbarrier and bulk-copy primitives (PTX ISA 8.x; sm_90 and later).
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase of the given parity to complete; gives up after `limit` polls (the error
// word is then set to VSHE_E_TIMEOUT) or once the error word is set by another thread.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity, unsigned long long limit, int32_t *err) {
  unsigned long long spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (++spins > limit) { atomicExch(err, VSHE_E_TIMEOUT_DEV); return false; }
    if ((spins & 63) == 0 && *((volatile int32_t *)err) != 0) return false;
    if (spins > 16) __nanosleep(64);
  }
  return true;
}
// The same for a whole warp, whose lanes all learn the same outcome: what follows a failed wait (barriers
// of the CTA, warp-wide instructions) must not find the warp split.  (One poll and a vote first, the loop
// out of the way: the local sweeps take 0.4 % longer than with lanes that decide alone, with a vote after
// the loop 2.8 %.)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, unsigned parity, unsigned long long limit, int32_t *err) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit, err));
}
// Waits for a phase regardless of the error word, at most kDrainPolls polls: copies in flight
// complete within microseconds, and shared memory must not be released under them.
constexpr unsigned long long kDrainPolls = 1ull << 24;
__device__ __forceinline__ void mbar_drain(uint64_t *bar, unsigned parity) {
  for (unsigned long long spins = 0; !mbar_try_wait(bar, parity) && spins < kDrainPolls; ++spins)
    if (spins > 16) __nanosleep(64);
}
// Bulk copy (the untiled TMA form) of `bytes` from global memory into this CTA's shared memory;
// completion is counted on the mbarrier.  Source, destination and size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Asynchronous copy of 8 bytes into shared memory, and the wait for the thread's own copies.
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Barrier of the consumer warps only (named barrier 1; the producer warp does not take part).
__device__ __forceinline__ void consumers_sync(int nthreads) { asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory"); }

}  // namespace vshe
