// The grid barrier of the persistent kernels.
#ifndef B2VM_GRID_BARRIER_CUH_
#define B2VM_GRID_BARRIER_CUH_

#include "dev_common.cuh"

namespace b2 {

// Grid-wide barrier over the n_lanes co-resident CTAs. Returns false when the
// wait was abandoned (budget exhausted here or abort raised by another lane).
// One counter that only grows, modulo 2^32: a lane adds itself with a release reduction and polls the counter until it stands at
// `target`, n_lanes more per barrier (differences only, so the wrap is no event). A launch counts from where the
// last one left off, which lane 0 notes on its way out, when every lane has read the old note. (Worked out from the counter
// itself, as its last multiple of n_lanes, it was wrong after 2^32 arrivals: 29 M barriers of 148 lanes.)
// What is not needed at every barrier stays out of this code: it is fetched anew every time, and two loads and a branch for
// the first barrier cost each of them 0.27 us.
// 1.15 us per barrier on 148 lanes (a counter and a generation word, both read and written by every lane: 1.77 us; a
// release line per lane: 1.73 us).
// Ordering: the CTA barrier makes the lane's stores visible to thread 0, whose release arrival publishes them (release is
// cumulative); the acquire load that closes the wait synchronises with every arrival before it (each addition continues
// the release sequences of the ones before), and the closing CTA barrier carries that to the lane's other threads.
// The last warp runs `meanwhile` under the wait.
template <typename F>
__device__ __forceinline__ bool grid_barrier(const Lane &L, uint32_t barrier_index, unsigned long long t_start, uint32_t &target,
                                             F meanwhile) {
  const KParams &P = *L.P;
  DSync *s = P.sync;
  __syncthreads();
  bool ok = true;
  if (L.tid == 0) {
    if (P.lane_ts && barrier_index < kPhaseSlots) P.lane_ts[L.lane * kLaneTsSlots + 2u + barrier_index] = globaltimer_ns();
    red_release_gpu_add(&s->arrive, 1u);
    target += P.n_lanes;
    uint32_t spins = 0;
    unsigned long long t0 = 0;
    while (static_cast<int32_t>(ld_relaxed_gpu(&s->arrive) - target) < 0) {
      if ((++spins & 63u) == 0u) {
        if (ld_relaxed_gpu(&s->abort)) { ok = false; break; }
        if (t0 == 0ull) t0 = globaltimer_ns();
        nanosleep_ns(64);
        if (globaltimer_ns() - t0 > P.wait_budget_ns) {
          set_status(P, kStBarrierTimeout, L.lane, barrier_index, 0u);
          ok = false;
          break;
        }
      }
    }
    ld_acquire_gpu(&s->arrive);
    // when the phase ended for everybody: the barrier's release as lane 0 sees it
    if (L.lane == 0 && barrier_index < kPhaseSlots) s->phase_ns[barrier_index] = globaltimer_ns() - t_start;
  } else if (L.tid >= L.nthr - kWarp) {
    meanwhile();
  }
  return __syncthreads_and(ok) != 0;
}

// Thread 0, as the launch begins: `target` before the first barrier. Behind a launch that failed the counts mean nothing: one
// that is not reached, so that the first wait finds the abort flag.
__device__ __forceinline__ uint32_t grid_barrier_base(const KParams &P) {
  return ld_relaxed_gpu(&P.sync->base) + (ld_relaxed_gpu(&P.sync->abort) ? 1u << 30 : 0u);
}
// Lane 0's thread 0, at the end of a launch that passed `barriers` barriers.
__device__ __forceinline__ void grid_barrier_done(const KParams &P, uint32_t barriers, uint32_t target) {
  if (barriers) P.sync->base = target;
}

}  // namespace b2
#endif
