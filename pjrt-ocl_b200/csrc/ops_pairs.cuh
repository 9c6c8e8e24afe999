// All-pairs accelerations (kTopPairs): the re-planner's form of the tile ops
//   d_ij = x_j - x_i;  r2 = rowsum(d * d);  w = m_j (r2 s + t)^-1.5;  out_i = sum_j w_ij d_ij
// which as bytecode is six to eight tile ops over (n, n) and (n, n, 3) tensors (1.3 GB per
// evaluation at n = 4096, 650 us). Here nothing of size n^2 exists: positions and masses sit in
// shared memory as float4, a thread keeps NI bodies i and their sums in registers and walks the
// j's of its slice.
//
// Bound: 18.8 us per evaluation of 4096 bodies in a loop of them (40 evaluations 763 us): 10.4 the pair loop - 7-8 of FP32 issue by count
// (16.8 M pairs of ~16 instructions on 148 SMs) beside 3.6 of square roots -, 3 the staging of all bodies, 1.2 the grid barrier, the
// rest sums, tail and set-up. Issue is 45 % active; barriers, of the lane and of the grid, are the top stall.
//
// Split: a lane owns bodies [lo, hi). Its 16 warps form `groups` i-groups (NI bodies each, all 32
// lanes of a warp the same ones) x 16 / groups j-slices; groups x NI is the smallest cover of the
// lane's bodies. Lane k of a warp takes j = k, k + 32, ... of the slice (conflict-free 16-byte reads,
// NI pairs per read); sums meet by shuffles, then across the slices in shared memory, in a fixed order.
// The roundings per pair are those of the separate ops up to the reciprocal square root, which is the
// hardware approximation with one Newton step (relative error ~1e-7); the sums are f32 in another order.
//
// The elementwise tail (the Runge-Kutta combinations that only need the lane's own rows) runs at the
// end on the lane's elements: one thread per element does all of them, so it needs no barrier.
#ifndef B2VM_OPS_PAIRS_CUH_
#define B2VM_OPS_PAIRS_CUH_

#include "dev_common.cuh"
#include "plan_format.h"
#include "ops_ew.cuh"

namespace b2 {

constexpr uint32_t kPairsChunk = 4096;                                   // bodies staged at a time (64 KB)
constexpr uint32_t kPairsMaxNi = 8;                                      // bodies per thread
constexpr uint32_t kPairsRows = 16 * kPairsMaxNi;                        // bodies of a lane worked on at a time
constexpr uint32_t kPairsJ = kSmemSys;                                   // float4 x, y, z, m
constexpr uint32_t kPairsPart = kPairsJ + kPairsChunk * 16u;             // partial sums [slice][body][3]
constexpr uint32_t kPairsExt = kPairsPart + kPairsRows * 3u * 4u;        // tail operands from memory [op][a, b][element]
constexpr uint32_t kPairsVal = kPairsExt + kPairTailMax * 2u * kPairsRows * 3u * 4u;   // the sum and the tail's results [1 + op][element]
static_assert(kPairsVal + (kPairTailMax + 1u) * kPairsRows * 3u * 4u <= 226u * 1024u, "fits the lane's shared memory");

// 1 / sqrt(a) by the special-function unit (flushes denormals; relative error ~2^-22).
__device__ __forceinline__ float fast_rsqrt(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

// The smaller of two, a NaN if either is one.
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int NI, bool UNIT>
static __device__ __noinline__ void pairs_run(const Lane &L, const DPairs &p, const float *pos, const float *mass, uint32_t lo, uint32_t hi,
                                              uint32_t groups) {
  const KParams &P = *L.P;
  float4 *sj = reinterpret_cast<float4 *>(L.smem + kPairsJ);
  float *part = reinterpret_cast<float *>(L.smem + kPairsPart);
  float *ext = reinterpret_cast<float *>(L.smem + kPairsExt), *val = reinterpret_cast<float *>(L.smem + kPairsVal);
  const uint32_t w = L.tid / kWarp, lane = L.tid % kWarp, nw = L.nthr / kWarp;
  const uint32_t slices = nw / groups, grp = w % groups, slice = w / groups;
  const uint32_t i0 = lo + grp * NI, elems = 3u * (hi - lo), n_tail = p.n_tail;
  const float as = p.s, at = p.t;
  float px[NI], py[NI], pz[NI], ax[NI], ay[NI], az[NI];
#pragma unroll
  for (int k = 0; k < NI; ++k) {
    const uint32_t i = min(i0 + k, p.n - 1u);
    px[k] = pos[3u * i]; py[k] = pos[3u * i + 1u]; pz[k] = pos[3u * i + 2u];
    ax[k] = ay[k] = az[k] = 0.0f;
  }
  const bool wide = ((reinterpret_cast<uintptr_t>(pos) | reinterpret_cast<uintptr_t>(mass)) & 15u) == 0u;
  for (uint32_t c0 = 0; c0 < p.n; c0 += kPairsChunk) {
    const uint32_t cn = min(kPairsChunk, p.n - c0);
    __syncthreads();
    const uint32_t quads = wide ? cn / 4u : 0u;
    for (uint32_t g = L.tid; g < quads; g += L.nthr) {          // four bodies by four 16-byte loads
      const float4 *q = reinterpret_cast<const float4 *>(pos + 3u * static_cast<size_t>(c0)) + 3u * g;
      const float4 a = q[0], b = q[1], c = q[2], m = reinterpret_cast<const float4 *>(mass + c0)[g];
      sj[4u * g] = make_float4(a.x, a.y, a.z, m.x);
      sj[4u * g + 1u] = make_float4(a.w, b.x, b.y, m.y);
      sj[4u * g + 2u] = make_float4(b.z, b.w, c.x, m.z);
      sj[4u * g + 3u] = make_float4(c.y, c.z, c.w, m.w);
    }
    for (uint32_t j = 4u * quads + L.tid; j < cn; j += L.nthr) {
      const float *q = pos + 3u * static_cast<size_t>(c0 + j);
      sj[j] = make_float4(q[0], q[1], q[2], mass[c0 + j]);
    }
    if (c0 == 0u) {                                             // the tail's operands from memory, a warp each, under the pair loop
      for (uint32_t oa = w; oa < 2u * n_tail; oa += nw) {
        const DPairTail &tl = p.tail[oa >> 1];
        const BufRef r = (oa & 1u) ? tl.b : tl.a;
        if (((oa & 1u) ? tl.b_src : tl.a_src) != 0u || !r) continue;
        const float *src = reinterpret_cast<const float *>(resolve(P, r)) + 3u * static_cast<size_t>(lo);
        for (uint32_t e = lane; e < elems; e += kWarp) cp_async_4_zfill(smem_addr(ext + oa * (kPairsRows * 3u) + e), src + e, 4u);
      }
    }
    __syncthreads();
    const uint32_t j_lo = cn * slice / slices, j_hi = cn * (slice + 1u) / slices;
#pragma unroll 2
    for (uint32_t j = j_lo + lane; j < j_hi; j += kWarp) {
      const float4 q = sj[j];
      const float m15 = 1.5f * q.w;
#pragma unroll
      for (int k = 0; k < NI; ++k) {
        const float dx = q.x - px[k], dy = q.y - py[k], dz = q.z - pz[k];
        // (a squared distance beyond f32 weighs nothing: infinity times the root's zero would be a NaN)
        const float a = min_nan(UNIT ? fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, at))) : fmaf(fmaf(dz, dz, fmaf(dy, dy, dx * dx)), as, at), 3.402823466e38f);
        const float r = fast_rsqrt(a), r2 = r * r;
        // a^-1.5 = r^3 (1 + 1.5 (1 - a r^2) + ...): first-order correction of the approximate root
        const float wj = (r2 * r) * fmaf(fmaf(-a, r2, 1.0f), m15, q.w);
        ax[k] = fmaf(wj, dx, ax[k]);
        ay[k] = fmaf(wj, dy, ay[k]);
        az[k] = fmaf(wj, dz, az[k]);
      }
    }
  }
  // The warp's sums: of 24 values (eight bodies) a lane hands on half, then half of that, then half again; two whole steps are left,
  // and lanes 4 k .. 4 k + 3 hold body k. (One value at a time the 21 of seven bodies took 1900 cycles.)
  const uint32_t cover = groups * NI;
  {
    float v[24] = {};
#pragma unroll
    for (int k = 0; k < NI; ++k) { v[3 * k] = ax[k]; v[3 * k + 1] = ay[k]; v[3 * k + 2] = az[k]; }
#pragma unroll
    for (int h = 12, o = 16; h >= 3; h /= 2, o /= 2) {
      const bool up = (lane & static_cast<uint32_t>(o)) != 0u;
#pragma unroll
      for (int k = 0; k < 12; ++k)
        if (k < h) {
          const float send = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
          v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    const uint32_t k = lane >> 2;                 // 4 b4 + 2 b3 + b2
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      v[e] += __shfl_xor_sync(0xffffffffu, v[e], 2);
      v[e] += __shfl_xor_sync(0xffffffffu, v[e], 1);
    }
    if ((lane & 3u) == 0u && k < static_cast<uint32_t>(NI)) {
      float *o = part + (static_cast<size_t>(slice) * cover + grp * NI + k) * 3u;
      o[0] = v[0]; o[1] = v[1]; o[2] = v[2];
    }
  }
  cp_async_wait_all();
  __syncthreads();
  float *out = reinterpret_cast<float *>(resolve(P, p.out));
  for (uint32_t e = L.tid; e < elems; e += L.nthr) {
    float s = 0.0f;
    for (uint32_t c = 0; c < slices; ++c) s += part[static_cast<size_t>(c) * cover * 3u + e];
    const size_t row = 3u * static_cast<size_t>(lo) + e;
    val[e] = s;
    out[row] = s;
    for (uint32_t q = 0; q < n_tail; ++q) {
      const DPairTail &tl = p.tail[q];
      const float x = tl.a_src ? val[(tl.a_src - 1u) * (kPairsRows * 3u) + e] : ext[(q * 2u) * (kPairsRows * 3u) + e];
      const float y = tl.b_src ? val[(tl.b_src - 1u) * (kPairsRows * 3u) + e] : ext[(q * 2u + 1u) * (kPairsRows * 3u) + e];
      const float v = tl.sub == kAffine ? affine2(x, tl.s, tl.t) : tl.sub == kAdd ? __fadd_rn(x, y) : tl.sub == kSubt ? __fsub_rn(x, y)
                      : tl.sub == kMul ? __fmul_rn(x, y) : x;
      val[(q + 1u) * (kPairsRows * 3u) + e] = v;
      reinterpret_cast<float *>(resolve(P, tl.dst))[row] = v;
    }
  }
}

static __device__ __noinline__ void pairs_tiles(const Lane &L, const DTask &t, uint32_t tile_lo, uint32_t tile_hi) {
  const KParams &P = *L.P;
  const DPairs &p = *reinterpret_cast<const DPairs *>(planned_desc(L, t));
  const uint32_t hi = min(tile_hi, p.n);
  const float *pos = reinterpret_cast<const float *>(resolve(P, p.pos)), *mass = reinterpret_cast<const float *>(resolve(P, p.mass));
  for (uint32_t lo = tile_lo; lo < hi; lo += kPairsRows) {       // at most 16 groups of 8 at a time
    const uint32_t h = min(hi, lo + kPairsRows), ni = h - lo;
    // the (groups, NI) with the fewest idle slots; more groups (shorter loops of more bodies) only if they cover better
    uint32_t groups = 16u, best = 0xffffffffu;
    for (uint32_t g = 16u; g >= 1u; g >>= 1) {
      const uint32_t k = (ni + g - 1u) / g;
      if (k <= kPairsMaxNi && g * k <= best) { best = g * k; groups = g; }
    }
    switch ((ni + groups - 1u) / groups) {
#define B2_PAIRS(N)                                                      \
  if (p.s == 1.0f) pairs_run<N, true>(L, p, pos, mass, lo, h, groups);   \
  else pairs_run<N, false>(L, p, pos, mass, lo, h, groups);              \
  break;
      case 1: B2_PAIRS(1)
      case 2: B2_PAIRS(2)
      case 3: B2_PAIRS(3)
      case 4: B2_PAIRS(4)
      case 5: B2_PAIRS(5)
      case 6: B2_PAIRS(6)
      case 7: B2_PAIRS(7)
      default: B2_PAIRS(8)
#undef B2_PAIRS
    }
  }
}

}  // namespace b2
#endif
