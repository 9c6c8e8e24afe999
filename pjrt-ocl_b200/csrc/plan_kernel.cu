// The persistent kernel of the re-planned programs (replan.h): one CTA per lane walks its entries - tile entries of
// the re-planner's own ops, grid barriers, at most one counted loop at the top - and nothing else, so that what stands
// between a launch (or a barrier) and the first load of data is short: the lane's head (span, first entry, first task) is one
// read, the rest of its entries and the next task with its descriptor arrive in shared memory while something else waits.
// A wire program's tile ops and control flow are vm_kernel.cu's.
#include <cuda_runtime.h>

// Compiled once per entry of variants.h whose name starts with "plan", with -DB2_VARIANT=<name> -DB2_FAMILIES=<mask>.
#ifndef B2_FAMILIES
#define B2_FAMILIES 0xFFFFFFFFu
#define B2_VARIANT plan
#endif
#define B2_HAS(fam) (((B2_FAMILIES) & (fam)) != 0u)
#define B2_PASTE2(a, b) a##b
#define B2_PASTE(a, b) B2_PASTE2(a, b)
#define B2_SHORT 1

#include <cstring>
#include "dev_common.cuh"
#include "grid_barrier.cuh"
#if B2_HAS(0x200u)  // kFamFuse
#include "ops_fuse.cuh"
#endif
#if B2_HAS(0x400u)  // kFamPairs
#include "ops_pairs.cuh"
#endif
#if B2_HAS(0x800u)  // kFamGemm
#include "ops_gemm.cuh"
#endif
#if B2_HAS(0x2000u) // kFamSgemm
#include "ops_sgemm.cuh"
#endif
#if B2_HAS(0x4000u) // kFamSkinny
#include "ops_skinny.cuh"
#endif
#if B2_HAS(0x40u)   // kFamFlash: the wire programs' attention
#include "ops_flash_tc.cuh"
#include "ops_flash.cuh"
#endif
#if B2_HAS(0x02u)   // kFamMove: and their moves
#include "ops_move.cuh"
#endif

namespace b2 {
static_assert(kFamFuse == 0x200u && kFamPairs == 0x400u && kFamGemm == 0x800u && kFamSgemm == 0x2000u && kFamSkinny == 0x4000u && kFamFlash == 0x40u && kFamMove == 0x02u, "the literals in the #if lines above");

constexpr int kVmThreads = 512;
constexpr uint32_t kNoPc = 0xFFFFFFFFu;
static_assert(kSmemEntries + kSmemEntriesMax * sizeof(DEntry) <= static_cast<uint32_t>(kSmemDesc) &&
              kSmemDesc + kSmemDescMax <= static_cast<uint32_t>(kSmemSys), "fits the interpreter's part of the shared memory");

// One warp: copies a planned op's descriptor, `words` = lane t's word of its task (t < 24).
__device__ __forceinline__ void stage_desc(const Lane &L, uint32_t words, uint32_t t) {
  const uint32_t desc = __shfl_sync(0xffffffffu, words, offsetof(DTask, desc) / 4u);
  const uint32_t bytes = __shfl_sync(0xffffffffu, words, offsetof(DTask, desc_bytes) / 4u);
  if (bytes == 0u || bytes > kSmemDescMax) return;
  const uint4 *src = reinterpret_cast<const uint4 *>(L.P->desc + desc);
#pragma unroll 4
  for (uint32_t i = t; i < bytes / 16u; i += 32u) reinterpret_cast<uint4 *>(L.smem + kSmemDesc)[i] = src[i];
  if (t == 0u) *reinterpret_cast<uint32_t *>(L.smem + kSmemNextDesc) = desc;
}

#define B2_PLAN_KERNEL B2_PASTE(b2_, B2_VARIANT)
__global__ void __launch_bounds__(kVmThreads, 1) B2_PLAN_KERNEL(const __grid_constant__ KParams P, const uint32_t smem_bytes) {
  B2_DYN_SMEM(smem);
  Lane L;
  L.P = &P;
  L.smem = smem;
  L.smem_bytes = smem_bytes;
  L.lane = blockIdx.x;
  L.tid = threadIdx.x;
  L.nthr = kVmThreads;
  const unsigned long long t_start = globaltimer_ns();
  if (P.lane_ts && L.tid == 0) P.lane_ts[L.lane * kLaneTsSlots] = t_start;
  uint32_t *next_pc = reinterpret_cast<uint32_t *>(smem + kSmemNextPc);
  uint32_t target = L.tid == 0 ? grid_barrier_base(P) : 0u;
  {
    const uint32_t *h = reinterpret_cast<const uint32_t *>(P.heads + L.lane);
    const uint32_t w = L.tid < sizeof(DHead) / 4u ? h[L.tid] : 0u;
    if (L.tid < 4u) reinterpret_cast<uint32_t *>(smem + kSmemRed)[L.tid] = w;
    else if (L.tid < 12u) reinterpret_cast<uint32_t *>(smem + kSmemEntries)[L.tid - 4u] = w;
    else if (L.tid < 36u) reinterpret_cast<uint32_t *>(smem + kSmemNextTask)[L.tid - 12u] = w;
    if (L.tid == 36u) { *next_pc = 0u; *reinterpret_cast<uint32_t *>(smem + kSmemNextDesc) = 0u; }
    __syncthreads();
  }
  const VmLane span = *reinterpret_cast<const VmLane *>(smem + kSmemRed);
  const DEntry *stream = P.entries + span.off;
  DEntry *ents = reinterpret_cast<DEntry *>(smem + kSmemEntries);
  if (L.tid < kWarp) {
    if (ents[0].task < kEntFor) stage_desc(L, L.tid < sizeof(DTask) / 4u ? reinterpret_cast<const uint32_t *>(smem + kSmemNextTask)[L.tid] : 0u, L.tid);
  } else if (L.tid >= 64u) {                       // the other entries, as many as fit
    const uint32_t n = min(span.count, kSmemEntriesMax) * 2u;
    for (uint32_t i = L.tid - 64u; i < n; i += L.nthr - 64u)
      if (i >= 2u) reinterpret_cast<uint4 *>(ents)[i] = reinterpret_cast<const uint4 *>(stream)[i];
  }
  __syncthreads();
  auto task_at = [&](uint32_t pc) { return pc < kSmemEntriesMax ? ents[pc].task : stream[pc].task; };
  // one warp, under a barrier wait: the task of the entry at `pc` and its descriptor
  auto stage_task = [&](uint32_t pc) {
    if (pc == kNoPc) return;
    const uint32_t t = L.tid & 31u, task = task_at(pc);
    if (task < kEntFor) {
      const uint32_t v = t < sizeof(DTask) / 4u ? reinterpret_cast<const uint32_t *>(P.tasks + task)[t] : 0u;
      if (t < sizeof(DTask) / 4u) reinterpret_cast<uint32_t *>(smem + kSmemNextTask)[t] = v;
      stage_desc(L, v, t);
      if (t == 0u) *next_pc = pc;
    }
  };

  uint32_t pc = 0, end = span.root_len, trips = 0, body = 0, ret = 0;   // trips: passes of the loop left, 0 outside it
  uint32_t barrier_i = 0;
  for (;;) {
    uint32_t then = kNoPc;            // a barrier is due; the entry after it
    bool bar = false;
    if (pc >= end) {
      if (trips == 0u) break;
      bar = true;                     // the pass is over
      if (--trips) { pc = body; }
      else { pc = ret; end = span.root_len; }
      then = pc < end ? pc : kNoPc;
    } else {
      const uint32_t task = task_at(pc);
      if (task == kEntBarrier) {
        bar = true;
        ++pc;
        then = pc < end ? pc : kNoPc;
      } else if (task == kEntFor) {
        const DEntry en = pc < kSmemEntriesMax ? ents[pc] : stream[pc];
        ret = pc + 1u;
        body = en.tile_lo;
        pc = body;
        end = body + en.tile_hi;
        trips = en.a;
        continue;
      }
    }
    if (bar) {
      if (!grid_barrier(L, barrier_i++, t_start, target, [&] { stage_task(then); })) break;
      continue;
    }
    const DEntry en = pc < kSmemEntriesMax ? ents[pc] : stream[pc];
    if (en.task != kEntNop) {
      __syncthreads();
      if (*next_pc != pc) {           // not staged: a second entry of a phase, or the first of a loop
        if (L.tid < sizeof(DTask) / 4u) reinterpret_cast<uint32_t *>(smem + kSmemNextTask)[L.tid] = reinterpret_cast<const uint32_t *>(P.tasks + en.task)[L.tid];
        if (L.tid == 0) *next_pc = kNoPc;
        __syncthreads();
      }
      const DTask &t = *reinterpret_cast<const DTask *>(smem + kSmemNextTask);
      switch (t.op) {
#if B2_HAS(0x200u)
        case kTopFuseRows: fuse_rows_tiles(L, t, en.tile_lo, en.tile_hi); break;
#endif
#if B2_HAS(0x400u)
        case kTopPairs: pairs_tiles(L, t, en.tile_lo, en.tile_hi); break;
#endif
#if B2_HAS(0x800u)
        case kTopGemm: gemm_tiles(L, t, en.tile_lo, en.tile_hi); break;
#endif
#if B2_HAS(0x2000u)
        case kTopSgemm: sgemm_tiles(L, t, en.tile_lo, en.tile_hi); break;
#endif
#if B2_HAS(0x4000u)
        case kTopSkinny: skinny_tiles(L, t, en.tile_lo, en.tile_hi); break;
#endif
#if B2_HAS(0x40u)
        case kTopFlashAttn: {
          const DFlash &df = *reinterpret_cast<const DFlash *>(P.desc + t.desc);
          if (!(df.tc_mode && flash_tc_tiles(L, t, en.tile_lo, en.tile_hi))) flash_simt_tiles(L, t, en.tile_lo, en.tile_hi);
          break;
        }
#endif
#if B2_HAS(0x02u)
        case kTopGather: case kTopDynGather: move_tiles(L, t, en.tile_lo, en.tile_hi, false); break;
        case kTopScatter: case kTopDynScatter: move_tiles(L, t, en.tile_lo, en.tile_hi, true); break;
#endif
        default:
          if (L.tid == 0) set_status(P, kStBadOp, L.lane, en.task, t.op);
          break;
      }
    }
    ++pc;
  }
  if (P.lane_ts && L.tid == 0) P.lane_ts[L.lane * kLaneTsSlots + 1u] = globaltimer_ns();
  if (L.lane == 0 && L.tid == 0) {
    grid_barrier_done(P, barrier_i, target);
    P.sync->barriers = barrier_i;
    P.sync->device_ns = globaltimer_ns() - t_start;
  }
}

// ---- host-side launch glue (called from runtime.cc through the table in variants.h) ----
cudaError_t B2_PASTE(LaunchVm_, B2_VARIANT)(const KParams &params, uint32_t n_lanes, int threads, uint32_t smem_bytes,
                                            cudaStream_t stream, const void *keep_base, size_t keep_bytes) {
  void *args[2] = {const_cast<KParams *>(&params), &smem_bytes};
  if (threads != kVmThreads) return cudaErrorInvalidValue;
  const void *fn = reinterpret_cast<const void *>(&B2_PLAN_KERNEL);
  cudaLaunchAttribute attr[2];
  std::memset(attr, 0, sizeof(attr));
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  unsigned n_attr = 1;
  if (keep_base && keep_bytes) {        // the program's tables stay in the L2 set-aside between the phases
    attr[1].id = cudaLaunchAttributeAccessPolicyWindow;
    attr[1].val.accessPolicyWindow.base_ptr = const_cast<void *>(keep_base);
    attr[1].val.accessPolicyWindow.num_bytes = keep_bytes;
    attr[1].val.accessPolicyWindow.hitRatio = 1.0f;
    attr[1].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr[1].val.accessPolicyWindow.missProp = cudaAccessPropertyNormal;
    n_attr = 2;
  }
  // {grid, block, dynamic shared memory, stream, attributes, their count}
  cudaLaunchConfig_t cfg = {dim3(n_lanes), dim3(static_cast<unsigned>(threads)), smem_bytes, stream, attr, n_attr};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

// Co-resident CTAs of this build at `threads` per lane and `smem_bytes` of dynamic shared memory.
cudaError_t B2_PASTE(VmResidency_, B2_VARIANT)(int device, int threads, uint32_t smem_bytes, int *max_lanes) {
  if (threads != kVmThreads) return cudaErrorInvalidValue;
  const void *fn = reinterpret_cast<const void *>(&B2_PLAN_KERNEL);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_bytes));
  if (e != cudaSuccess) return e;
  int per_sm = 0, sms = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem_bytes);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  *max_lanes = per_sm * sms;
  return cudaSuccess;
}

}  // namespace b2
