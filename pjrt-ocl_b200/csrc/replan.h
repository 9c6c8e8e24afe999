// Re-plans a program for this device before its tables are built (loader.h).
//
// A VMProgram arrives as tile ops in barrier phases, cut over the lanes for a device where every
// tile op makes one pass over memory. The re-planner reads it back into a graph of tasks over
// buffers (the root walk, and the body of one counted loop), replaces groups of tasks by fused
// ops of this backend's own (format.h: kTopFuseRows, kTopPairs), orders what is left into as few
// phases as the data dependences allow, cuts every phase over all lanes of the device and places the
// remaining buffers anew. Results keep the roundings of every value that the program stores or
// hands on in a narrower type; sums may be taken in another order.
//
// A program keeps its schedule (loader.h: PlanGains) where the plan would make the same passes over memory, on the step
// interpreter. The re-planner leaves it alone (returns false) when nothing in it fuses, when it uses control flow other than one counted
// loop at the top, or when it was scheduled for half of the device or less.
#ifndef B2VM_REPLAN_H_
#define B2VM_REPLAN_H_

#include <cstdint>

#include "vmprog.h"

namespace b2 {

struct ReplanStats {
  uint32_t fused_rows = 0;   // row pipelines
  uint32_t pairs = 0;        // all-pairs evaluations
  uint32_t gemms = 0;        // matmuls with what followed them as store epilogue
  uint32_t absorbed = 0;     // tasks of the program that no longer exist
  uint32_t phases = 0;       // barrier phases of the new plan (root and loop body)
};

bool Replan(const VmProgram &p, uint32_t device_lanes, VmProgram *q, ReplanStats *st);

// Lists in the aux pool that the re-planner's own ops carry at p2: {n_reads, n_writes, reads, writes, payload}.
bool IsPlannedOp(uint32_t tile_op);
void PlannedLists(const VmProgram &p, const VmTask &t, const int32_t **reads, int *n_reads, const int32_t **writes, int *n_writes,
                  const int32_t **payload);

// Words before the steps in a kTopFuseRows payload: rows cols steps total+1 vec owners elements, and the phases of the schedule that
// it takes the place of.
constexpr int kFuseWords = 8;

// Words per product in a kTopGemm payload {n, total + 1, owner lanes, products}: M N K halves bn amn bmn adt a b a_ld b_ld a_off b_off
// epi qdt rdt s0 s1 gg res+1 out0+1 dt0 out1+1 dt1.
constexpr int kGemmWords = 25;

}  // namespace b2
#endif
