// Shared by the tensor-core tile ops: operand descriptors and bounded waits.
#ifndef B2VM_TC_COMMON_CUH_
#define B2VM_TC_COMMON_CUH_

#include "dev_common.cuh"

namespace b2 {

// Shared-memory matrix descriptor, 128-byte swizzle (layout type 2), descriptor version 1.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(lbo_bytes >> 4) << 16) |
         (static_cast<uint64_t>(sbo_bytes >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// Bounded wait that also gives up when another role of the lane failed.
// `backoff_ns`: sleep between polls - for waits that are expected to be long (the
// epilogue warps during the main loop), so they leave the issue slots to the producers.
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *failed,
                                        unsigned long long budget_ns, uint32_t backoff_ns = 0) {
  if (mbar_try_wait_parity(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
    for (int i = 0; i < 32; ++i) {
      if (mbar_try_wait_parity(bar, parity)) return true;
      if (backoff_ns) nanosleep_ns(backoff_ns);
    }
    if (*failed) return false;
    if (globaltimer_ns() - t0 > budget_ns) { *failed = 1u; return false; }
  }
}

// A whole warp waits, but only lane 0 polls: the other lanes sit at the warp
// barrier without taking issue slots from the warps that have work. Every lane
// gets lane 0's outcome (so the warp stays together when a wait ran out), and the
// warp barrier orders lane 0's acquire before the other lanes' later accesses.
__device__ __forceinline__ bool tc_wait_warp(uint64_t *bar, uint32_t parity, volatile uint32_t *failed,
                                             unsigned long long budget_ns, uint32_t backoff_ns = 0) {
  uint32_t ok = 1u;
  if ((threadIdx.x & 31u) == 0u) ok = tc_wait(bar, parity, failed, budget_ns, backoff_ns) ? 1u : 0u;
  return __shfl_sync(0xffffffffu, ok, 0) != 0u;
}

// The same with every lane polling and the warp in step throughout: for a warp whose elected lane issues products and commits.
// With lane 0 polling for the others a long wait (operands and code out of L2) now and then cost the warp a commit of its
// elected lane, and the lane's stages stood still until the wait ran out: 33 x 4096 by 4096 x 16000 within 40 launches.
__device__ __forceinline__ bool tc_wait_uniform(uint64_t *bar, uint32_t parity, volatile uint32_t *failed, unsigned long long budget_ns) {
  if (__all_sync(0xffffffffu, mbar_try_wait_parity(bar, parity))) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
    for (int i = 0; i < 32; ++i)
      if (__all_sync(0xffffffffu, mbar_try_wait_parity(bar, parity))) return true;
    const bool stop = *failed != 0u, late = globaltimer_ns() - t0 > budget_ns;
    if (__any_sync(0xffffffffu, stop || late)) {
      *failed = 1u;
      return false;
    }
  }
}

// The thread that fills a ring of stages, at its end: waits until the products have read what it filled last (`it` stages so
// far). Their commits arrive on the stages' empty barriers, which nobody else waits for: one still under way when the barriers
// are invalidated, or when the CTA is gone, is a fault.
__device__ __forceinline__ void tc_drain(uint64_t *empty, uint32_t stages, uint32_t it, volatile uint32_t *failed, unsigned long long budget_ns) {
  for (uint32_t k = 0; k < stages; ++k, ++it)
    if (!tc_wait(&empty[it % stages], ((it / stages) & 1u) ^ 1u, failed, budget_ns)) return;
}

}  // namespace b2
#endif
