// Asynchronous global -> shared copies for sm_100a: 1-D bulk copies (TMA
// engine, completion counted in bytes on an mbarrier) and the mbarrier
// operations around them.  No cluster multicast is used anywhere: every copy
// lands in the issuing CTA's own shared memory.
//
// Every wait here is bounded by wall time (%globaltimer); a wait that runs
// out returns false and the caller records the failure and leaves cleanly.
#pragma once
#include <cstdint>

#include "waits.cuh"

namespace a2d {

// how long one try of a wait may suspend its warp (it wakes when the phase completes)
constexpr uint32_t kSuspendNs = 100000;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// makes initialised mbarriers visible to the asynchronous (bulk copy) proxy
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// one arrival that also announces `bytes` of bulk-copy data for the current phase
__device__ __forceinline__ void mbar_arrive_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
      : "memory");
  return ok != 0;
}

// whether the phase of parity `parity` is complete, without waiting
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// waits for the phase of parity `parity` to complete; false after kWaitLimitNs.  By lanes each for
// itself, which vote on the verdicts before they go different ways
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  return bounded_wait([&] { return mbar_try_wait(bar, parity); }, global_ns, [](bool b) { return b; });
}

// a verdict of the whole warp
__device__ __forceinline__ bool warp_all(bool b) { return __all_sync(0xffffffffu, b); }

// the same by a whole warp, with one verdict
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
  return bounded_wait([&] { return mbar_try_wait(bar, parity); }, global_ns, warp_all);
}

// bulk copy of `bytes` (multiple of 16, both addresses 16-byte aligned) into
// this CTA's shared memory; completion is signalled on `bar` as transaction bytes
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// L2 policy for data a kernel streams once (factor blocks, Krylov basis runs):
// evicted first, so that the smaller vectors the kernel and its successors
// re-read stay in L2
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// bulk_load with an L2 cache policy for the source lines
__device__ __forceinline__ void bulk_load_hint(void* dst, const void* src, uint32_t bytes, uint64_t* bar,
                                               uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

// one plain arrival (no transaction bytes)
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace a2d
