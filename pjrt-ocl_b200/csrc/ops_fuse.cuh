// Fused row pipelines (kTopFuseRows): what the re-planner makes of neighbouring row-local
// tile ops - elementwise chains, LAYERNORM_SEG / SOFTMAX_SEG, row reductions and the scalar
// work on their results, broadcasts of per-row and per-column vectors, and the full sum of a
// value on the way. A group of T threads owns a row, holds it in registers from the first load
// to the last store (G groups of 4 elements per thread) and interprets the step list of the
// task (format.h: DFuStep); one dispatch covers all of a thread's elements.
//
// Bound: HBM for long f32 rows, instruction issue for 16-bit ones (the chain LayerNorm, x gamma
// + beta, GELU, softmax costs ~30 instructions per element whatever the storage type). As
// separate ops every intermediate went through memory: the chain moved 7 x the tensor, now 2 x.
//
// Layout: with cols % 4 == 0 element e of group g is column (g T + t) 4 + e (16-byte accesses for
// f32, 8-byte for 16-bit types, both fully coalesced); other rows start at any alignment and
// take column (4 g + e) T + t, one element per access, still coalesced. The dense loads of
// the NEXT row are started before the current row's steps: as per-thread asynchronous copies
// into the thread's own staging slots (no barrier needed to read them back), or, for accesses
// too narrow for those, as L2 prefetches. Column vectors are staged once per entry.
#ifndef B2VM_OPS_FUSE_CUH_
#define B2VM_OPS_FUSE_CUH_

#include "dev_common.cuh"
#include "plan_format.h"
#include "ops_ew.cuh"

namespace b2 {

constexpr uint32_t kFuseSteps = kSmemSys;                                   // resolved steps
constexpr uint32_t kFuseSlots = kFuseSteps + kFuMaxSteps * 32u;             // group reduction slots: 8 groups x 64 floats (warps alone need none)
constexpr uint32_t kFuseData = kFuseSlots + 8u * 64u * 4u;                  // staged vectors and rows
static_assert(kFuseData % 128u == 0u, "staging is 128-byte aligned");
static_assert(kFuseData + 128u <= kLaneSmemBytes - kPlanStageBytes, "what the loader counts on (plan_format.h)");

struct FuStep { uint32_t code, dt; float s, t; uint8_t *ptr; uint32_t reg, slot; };
static_assert(sizeof(FuStep) == 32, "same size as on the wire");

// Eight 16-bit values out of a 16-byte word.
__device__ __forceinline__ void unpack8(const uint4 &u, uint32_t dt, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = dt == kBF16 ? __uint_as_float(w[i] << 16) : f16_bits_to_f32(w[i] & 0xffffu);
    f[2 * i + 1] = dt == kBF16 ? __uint_as_float(w[i] & 0xffff0000u) : f16_bits_to_f32(w[i] >> 16);
  }
}

// 1 / x and 1 / sqrt(x) to about one unit in the last place, for normal x: the special-function unit's approximation and
// one Newton step. Used where the correctly rounded forms would put a subroutine call (their slow path) into the step
// loop, which makes the compiler keep a thread's elements where the call wants them and move them around every step.
__device__ __forceinline__ float rcp_nr(float x) {
  const float r = fast_rcp(x);
  const float e = fmaf(-x, r, 1.0f);
  return x > 1.0e-37f && x < 1.0e37f ? fmaf(r, e, r) : r;
}
__device__ __forceinline__ float rsqrt_nr(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float e = fmaf(-x * r, r, 1.0f);
  return x > 1.0e-37f && x < 1.0e37f ? fmaf(0.5f * r, e, r) : r;
}

// The same for a mean square that may be denormal (a norm without an epsilon): scaled, where the approximation would flush it.
// (Layer norms, whose variance is a difference that loses such numbers, keep the shorter form: 98 us for 101 at 8192 x 4096 f32.)
__device__ __forceinline__ float rsqrt_nr_tiny(float x) {
  const bool tiny = x < 1.0e-37f;
  const float r = rsqrt_nr(x * (tiny ? 0x1p+64f : 1.0f));
  return tiny ? r * 0x1p+32f : r;
}

// d/dz of tanh-GELU, 0.5 (1 + t) + 0.5 z (1 - t^2) u' with t = tanh(u), u = k (z + 0.044715 z^3), u' = k + c z^2: with
// e = exp(2u) and r = 1 / (1 + e) that is 0.5 (1 + t) = e r and 1 - t^2 = 4 e r^2, so e r (1 + 2 z r u'): one exponential
// and one reciprocal, no cancellation. c = 3 x 0.7978845608 x 0.044715 as the program rounds it.
__device__ __forceinline__ float gelu_grad(float z, float c) {
  const float z2 = z * z;
  const float a = fminf(z * fmaf(z2, 2.3022082f * 0.044715f, 2.3022082f), 100.0f);      // 2 u log2(e)
  const float e = fast_ex2(a), r = fast_rcp(1.0f + e);
  return (e * r) * fmaf(2.0f * z * r, fmaf(z2, c, 0.7978845608f), 1.0f);
}

// Reduce two values over the T threads of a row group (a warp, or whole warps). `slot` = 64 floats of the group: the two
// halves are used in turn (`turn`), so one barrier per reduction is enough - the next one's orders this one's reads
// before the half is written again.
template <typename F>
__device__ __forceinline__ float2 fuse_group_reduce2(float v, float v2, F f, float *slot, uint32_t T, uint32_t gi, uint32_t gl, uint32_t &turn) {
#pragma unroll
  for (int o = kWarp / 2; o > 0; o >>= 1) {
    v = f(v, __shfl_xor_sync(0xffffffffu, v, o));
    v2 = f(v2, __shfl_xor_sync(0xffffffffu, v2, o));
  }
  if (T == static_cast<uint32_t>(kWarp)) return make_float2(v, v2);
  float2 *h = reinterpret_cast<float2 *>(slot) + (turn ? 16 : 0);
  turn ^= 1u;
  if ((gl & 31u) == 0u) h[gl >> 5] = make_float2(v, v2);
  bar_sync(1 + static_cast<int>(gi), static_cast<int>(T));
  float2 r = h[0];
  for (uint32_t w = 1; w < (T >> 5); ++w) { r.x = f(r.x, h[w].x); r.y = f(r.y, h[w].y); }
  return r;
}
template <typename F>
__device__ __forceinline__ float fuse_group_reduce(float v, F f, float *slot, uint32_t T, uint32_t gi, uint32_t gl, uint32_t &turn) {
  v = warp_reduce(v, f);
  if (T == static_cast<uint32_t>(kWarp)) return v;
  float2 *h = reinterpret_cast<float2 *>(slot) + (turn ? 16 : 0);
  turn ^= 1u;
  if ((gl & 31u) == 0u) h[gl >> 5].x = v;
  bar_sync(1 + static_cast<int>(gi), static_cast<int>(T));
  float r = h[0].x;
  for (uint32_t w = 1; w < (T >> 5); ++w) r = f(r, h[w].x);
  return r;
}

// A full sum shared by `owners` lanes: every lane leaves its total, the last to arrive adds
// them in lane order. `slot` picks one of the counters of the scratch. All threads call.
__device__ __forceinline__ void fuse_full_sum(const Lane &L, float v, float *dst, uint32_t slot, uint32_t owners) {
  const KParams &P = *L.P;
  RedScratch *sc = reinterpret_cast<RedScratch *>(P.scratch);
  v = block_reduce(L, v, [](float a, float c) { return a + c; }, 0.0f);
  float *tot = reinterpret_cast<float *>(&sc->total[static_cast<size_t>(2u + slot) * P.n_lanes]);
  uint32_t *flag = reinterpret_cast<uint32_t *>(L.smem + kSmemFlag) + 1;
  if (L.tid == 0) {
    tot[2u * L.lane] = v;
    tot[2u * L.lane + 1u] = 1.0f;             // this lane took part
    *flag = atom_add_acq_rel_gpu(&sc->pad[slot], 1u) == owners - 1u ? 1u : 0u;
  }
  __syncthreads();
  if (*flag) {
    float s = 0.0f;
    if (L.tid < kWarp) {
      for (uint32_t l = L.tid; l < P.n_lanes; l += kWarp) {
        volatile float *q = tot + 2u * l;
        if (q[1] != 0.0f) { s += q[0]; q[1] = 0.0f; }
      }
      s = warp_reduce(s, [](float a, float c) { return a + c; });
      if (L.tid == 0) {
        *dst = s;
        st_relaxed_gpu(&sc->pad[slot], 0u);
      }
    }
  }
  __syncthreads();
}

// RARE: with the steps whose code holds subroutine calls (division, logarithms, ...) compiled in.
template <int G, bool VEC, bool RARE>
static __device__ __noinline__ float fuse_rows_run(uint32_t tid, uint32_t nthr, uint32_t T, uint32_t lo, uint32_t hi, uint32_t cols,
                                                   uint32_t nsteps, uint32_t stage_off, uint32_t stage_slots, uint32_t n_loads, uint32_t n_elems) {
  B2_DYN_SMEM(sm);
  const FuStep *steps = reinterpret_cast<const FuStep *>(sm + kFuseSteps);
  const uint32_t *loads = reinterpret_cast<const uint32_t *>(sm + kSmemChain);     // which steps are dense loads
  const uint32_t gi = tid / T, gl = tid % T, ng = nthr / T;
  float *slot = reinterpret_cast<float *>(sm + kFuseSlots) + (T > 32u ? gi * 64u : 0u);
  uint32_t turn = 0;
  // this thread's staging: [2 buffers][slots][G] 16-byte words, word index interleaved over the threads
  uint8_t *stage = sm + stage_off;
  auto stage_at = [&](uint32_t buf, uint32_t sl, int g) {
    return stage + ((static_cast<size_t>(buf * stage_slots + sl) * G + g) * nthr + tid) * 16u;
  };
  auto col_of = [&](int g, int e) -> uint32_t {
    return VEC ? ((static_cast<uint32_t>(g) * T + gl) << 2) + e : (static_cast<uint32_t>(4 * g + e)) * T + gl;
  };
  // This thread's groups (VEC) or elements inside the row: the first `nv`, since columns ascend.
  auto valid = [&](uint32_t c) { return VEC ? (c > gl * 4u ? (c - gl * 4u + 4u * T - 1u) / (4u * T) : 0u) : (c > gl ? (c - gl + T - 1u) / T : 0u); };
  const uint32_t last_row = (n_elems - 1u) / cols, last_cols = n_elems - last_row * cols;
  const uint32_t nv_all = valid(cols), nv_last = valid(last_cols);
  auto start_loads = [&](uint32_t row, uint32_t buf) {     // the dense loads of `row`
    const uint32_t nv = row == last_row ? nv_last : nv_all;
    for (uint32_t si = 0; si < n_loads; ++si) {
      const FuStep &st = steps[loads[si]];
      const uint32_t esz = dt_size(st.dt);
      const uint8_t *q = st.ptr + static_cast<size_t>(row) * cols * esz;
      if (VEC && st.slot != kFuNoSlot) {
        uint32_t d = smem_addr(stage_at(buf, st.slot, 0));
        q += static_cast<size_t>(gl) * 4u * esz;
        const uint32_t qs = T * 4u * esz;
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if (static_cast<uint32_t>(g) < nv) {
            if (esz == 4u) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(q) : "memory");
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(q) : "memory");
          }
          d += nthr * 16u;
          q += qs;
        }
      } else {
        const uint32_t nb = (row == last_row ? last_cols : cols) * esz;
        for (uint32_t b = gl * 128u; b < nb; b += T * 128u) prefetch_l2(q + b);
      }
    }
    cp_async_commit();
  };
  const float inv_cols = 1.0f / static_cast<float>(cols);
  float csum = 0.0f;
  uint32_t buf = 0;
  uint32_t row = lo + gi;
  if (row < hi) start_loads(row, 0u);
  for (; row < hi; row += ng) {
    float X[G][4], Y[G][4], S[kFuScalars];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int e = 0; e < 4; ++e) X[g][e] = Y[g][e] = 0.0f;
#pragma unroll
    for (int k = 0; k < kFuScalars; ++k) S[k] = 0.0f;
    cp_async_wait<0>();
    if (row + ng < hi) start_loads(row + ng, buf ^ 1u);
    const size_t rbase = static_cast<size_t>(row) * cols;
    const uint32_t nv = row == last_row ? nv_last : nv_all, row_cols = row == last_row ? last_cols : cols;
    const bool full = row_cols == 4u * T * G;

#define B2_FU_ALL(...)                             \
  _Pragma("unroll") for (int g = 0; g < G; ++g)    \
  _Pragma("unroll") for (int e = 0; e < 4; ++e) { __VA_ARGS__; }
#define B2_FU_IN(...)                              \
  if (full) { B2_FU_ALL(__VA_ARGS__) } else {      \
    _Pragma("unroll") for (int g = 0; g < G; ++g)  \
    _Pragma("unroll") for (int e = 0; e < 4; ++e) if (static_cast<uint32_t>(VEC ? g : 4 * g + e) < nv) { __VA_ARGS__; } }
    auto unpack4 = [](uint2 w, uint32_t dt, float (&R)[4]) {
      if (dt == kBF16) {
        R[0] = __uint_as_float(w.x << 16); R[1] = __uint_as_float(w.x & 0xffff0000u);
        R[2] = __uint_as_float(w.y << 16); R[3] = __uint_as_float(w.y & 0xffff0000u);
      } else {
        R[0] = f16_bits_to_f32(w.x & 0xffffu); R[1] = f16_bits_to_f32(w.x >> 16);
        R[2] = f16_bits_to_f32(w.y & 0xffffu); R[3] = f16_bits_to_f32(w.y >> 16);
      }
    };
    // consecutive elements starting at `q` (already at the row / vector start); staged rows come from shared memory
    auto load = [&](float (&R)[G][4], const uint8_t *q, uint32_t dt, uint32_t sl) {
      if (VEC) {
        if (sl != kFuNoSlot) {
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const uint8_t *w = stage_at(buf, sl, g);
            if (dt == kF32) {
              const float4 f = *reinterpret_cast<const float4 *>(w);
              R[g][0] = f.x; R[g][1] = f.y; R[g][2] = f.z; R[g][3] = f.w;
            } else {
              unpack4(*reinterpret_cast<const uint2 *>(w), dt, R[g]);
            }
          }
        } else if (dt == kF32) {
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const uint32_t c = col_of(g, 0);
            const float4 f = static_cast<uint32_t>(g) < nv ? *reinterpret_cast<const float4 *>(q + static_cast<size_t>(c) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            R[g][0] = f.x; R[g][1] = f.y; R[g][2] = f.z; R[g][3] = f.w;
          }
        } else {
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const uint32_t c = col_of(g, 0);
            unpack4(static_cast<uint32_t>(g) < nv ? *reinterpret_cast<const uint2 *>(q + static_cast<size_t>(c) * 2) : make_uint2(0u, 0u), dt, R[g]);
          }
        }
      } else if (dt == kF32) {
        B2_FU_ALL(const uint32_t c = col_of(g, e); R[g][e] = c < row_cols ? reinterpret_cast<const float *>(q)[c] : 0.0f)
      } else if (dt == kBF16) {
        B2_FU_ALL(const uint32_t c = col_of(g, e);
                  R[g][e] = c < row_cols ? __uint_as_float(static_cast<uint32_t>(reinterpret_cast<const uint16_t *>(q)[c]) << 16) : 0.0f)
      } else {
        B2_FU_ALL(const uint32_t c = col_of(g, e); R[g][e] = c < row_cols ? f16_bits_to_f32(reinterpret_cast<const uint16_t *>(q)[c]) : 0.0f)
      }
    };
    auto vec_load = [&](float (&R)[G][4], const FuStep &st) {
      // a staged vector sits at byte offset `slot` of the shared memory, in its storage type
      const uint8_t *q = st.slot != kFuNoSlot ? sm + st.slot : st.ptr;
      load(R, q, st.dt, kFuNoSlot);
    };
    auto quant = [&](float (&R)[G][4], uint32_t dt) {
      if (dt == kBF16) {
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const uint32_t w = cvt_bf16x2(R[g][e + 1], R[g][e]);
            R[g][e] = __uint_as_float(w << 16);
            R[g][e + 1] = __uint_as_float(w & 0xffff0000u);
          }
      } else if (dt == kF16) {
        B2_FU_ALL(R[g][e] = f16_bits_to_f32(f32_to_f16_bits(R[g][e])))
      }
    };
    auto add_f = [](float a, float c) { return a + c; };
    for (uint32_t si = 0; si < nsteps; ++si) {
      const FuStep &st = steps[si];
      switch (st.code) {
        case kFuLoadX: load(X, st.ptr + rbase * dt_size(st.dt), st.dt, st.slot); break;
        case kFuLoadY: load(Y, st.ptr + rbase * dt_size(st.dt), st.dt, st.slot); break;
        case kFuRowVecY: vec_load(Y, st); break;
        case kFuColVecY: { const float v = loadf(st.ptr, st.dt, row); B2_FU_ALL(Y[g][e] = v) break; }
        case kFuScalarY: { const float v = loadf(st.ptr, st.dt, 0); B2_FU_ALL(Y[g][e] = v) break; }
        case kFuStore: {
          uint8_t *q = st.ptr + rbase * dt_size(st.dt);
          if (VEC) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
              const uint32_t c = col_of(g, 0);
              if (static_cast<uint32_t>(g) < nv) {
                if (st.dt == kF32) *reinterpret_cast<float4 *>(q + static_cast<size_t>(c) * 4) = make_float4(X[g][0], X[g][1], X[g][2], X[g][3]);
                else if (st.dt == kBF16) *reinterpret_cast<uint2 *>(q + static_cast<size_t>(c) * 2) = make_uint2(cvt_bf16x2(X[g][1], X[g][0]), cvt_bf16x2(X[g][3], X[g][2]));
                else *reinterpret_cast<uint2 *>(q + static_cast<size_t>(c) * 2) =
                         make_uint2(f32_to_f16_bits(X[g][0]) | (f32_to_f16_bits(X[g][1]) << 16), f32_to_f16_bits(X[g][2]) | (f32_to_f16_bits(X[g][3]) << 16));
              }
            }
          } else if (st.dt == kF32) {
            B2_FU_IN(reinterpret_cast<float *>(q)[col_of(g, e)] = X[g][e])
          } else if (st.dt == kBF16) {
            B2_FU_IN(reinterpret_cast<uint16_t *>(q)[col_of(g, e)] = static_cast<uint16_t>(cvt_bf16x2(0.0f, X[g][e])))
          } else {
            B2_FU_IN(reinterpret_cast<uint16_t *>(q)[col_of(g, e)] = static_cast<uint16_t>(f32_to_f16_bits(X[g][e])))
          }
          break;
        }
        case kFuQuant: quant(X, st.dt); break;
        case kFuQuantY: quant(Y, st.dt); break;
        case kFuMovYX: B2_FU_ALL(Y[g][e] = X[g][e]) break;
        case kFuAdd: B2_FU_ALL(X[g][e] = __fadd_rn(X[g][e], Y[g][e])) break;
        case kFuMul: B2_FU_ALL(X[g][e] = __fmul_rn(X[g][e], Y[g][e])) break;
        case kFuSub: B2_FU_ALL(X[g][e] = __fsub_rn(X[g][e], Y[g][e])) break;
        case kFuRSub: B2_FU_ALL(X[g][e] = __fsub_rn(Y[g][e], X[g][e])) break;
        case kFuDiv: if constexpr (RARE) { B2_FU_ALL(X[g][e] = __fdiv_rn(X[g][e], Y[g][e])) } break;
        case kFuRDiv: if constexpr (RARE) { B2_FU_ALL(X[g][e] = __fdiv_rn(Y[g][e], X[g][e])) } break;
        case kFuMax: B2_FU_ALL(X[g][e] = np_max(X[g][e], Y[g][e])) break;
        case kFuMin: B2_FU_ALL(X[g][e] = np_min(X[g][e], Y[g][e])) break;
        case kFuAddS: { const float v = st.reg ? S[1] : S[0]; B2_FU_ALL(X[g][e] = __fadd_rn(X[g][e], v)) break; }
        case kFuMulS: { const float v = st.reg ? S[1] : S[0]; B2_FU_ALL(X[g][e] = __fmul_rn(X[g][e], v)) break; }
        case kFuSubS: { const float v = st.reg ? S[1] : S[0]; B2_FU_ALL(X[g][e] = __fsub_rn(X[g][e], v)) break; }
        case kFuDivS: if constexpr (RARE) { const float v = st.reg ? S[1] : S[0]; B2_FU_ALL(X[g][e] = __fdiv_rn(X[g][e], v)) } break;
        case kFuAffine: { const float s = st.s, t = st.t; B2_FU_ALL(X[g][e] = affine2(X[g][e], s, t)) break; }
        case kFuGelu: B2_FU_ALL(X[g][e] = gelu_tanh(X[g][e])) break;
        case kFuGeluGrad: B2_FU_ALL(X[g][e] = gelu_grad(X[g][e], st.s)) break;
        case kFuGeluGradY: B2_FU_ALL(Y[g][e] = gelu_grad(Y[g][e], st.s)) break;
        case kFuExp: if constexpr (RARE) { B2_FU_ALL(X[g][e] = expf(X[g][e])) } break;
        case kFuTanh: if constexpr (RARE) { B2_FU_ALL(X[g][e] = tanhf(X[g][e])) } break;
        case kFuNeg: B2_FU_ALL(X[g][e] = -X[g][e]) break;
        case kFuAbs: B2_FU_ALL(X[g][e] = fabsf(X[g][e])) break;
        case kFuSqrt: if constexpr (RARE) { B2_FU_ALL(X[g][e] = __fsqrt_rn(X[g][e])) } break;
        case kFuRsqrt: if constexpr (RARE) { B2_FU_ALL(X[g][e] = __fdiv_rn(1.0f, __fsqrt_rn(X[g][e]))) } break;
        case kFuLog: if constexpr (RARE) { B2_FU_ALL(X[g][e] = logf(X[g][e])) } break;
        case kFuRedSum: case kFuRedSumSq: {
          float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (st.code == kFuRedSum) { B2_FU_IN(a[e] += X[g][e]) }
          else { B2_FU_IN(a[e] = __fadd_rn(a[e], __fmul_rn(X[g][e], X[g][e]))) }
          const float v = fuse_group_reduce((a[0] + a[1]) + (a[2] + a[3]), add_f, slot, T, gi, gl, turn);
          if (st.reg) S[1] = v; else S[0] = v;
          break;
        }
        case kFuRedMax: {
          float v = -INFINITY;
          B2_FU_IN(v = np_max(v, X[g][e]))
          v = fuse_group_reduce(v, [](float a, float c) { return np_max(a, c); }, slot, T, gi, gl, turn);
          if (st.reg) S[1] = v; else S[0] = v;
          break;
        }
        case kFuSAffine: { const float v = affine2(st.reg ? S[1] : S[0], st.s, st.t); if (st.reg) S[1] = v; else S[0] = v; break; }
        case kFuSRsqrt: { const float v = rsqrt_nr_tiny(st.reg ? S[1] : S[0]); if (st.reg) S[1] = v; else S[0] = v; break; }
        case kFuLayerNorm: {
          float a[4] = {0.0f, 0.0f, 0.0f, 0.0f}, b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          B2_FU_IN(a[e] += X[g][e]; b[e] = fmaf(X[g][e], X[g][e], b[e]))
          const float2 r2 = fuse_group_reduce2((a[0] + a[1]) + (a[2] + a[3]), (b[0] + b[1]) + (b[2] + b[3]), add_f, slot, T, gi, gl, turn);
          const float s = r2.x, s2 = r2.y;
          const float inv_n = inv_cols;
          const float mu = s * inv_n;
          const float var = __fsub_rn(s2 * inv_n, __fmul_rn(mu, mu));
          const float rden = rsqrt_nr(__fadd_rn(var, st.s));
          B2_FU_ALL(X[g][e] = (X[g][e] - mu) * rden)
          break;
        }
        case kFuSoftmax: {
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          B2_FU_IN(mx[e] = fmaxf(mx[e], X[g][e]))            // a NaN still poisons the row through the sum
          const float m = fuse_group_reduce(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), [](float a, float c) { return fmaxf(a, c); }, slot, T, gi,
                                            gl, turn);
          float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          B2_FU_ALL(X[g][e] = fast_ex2((X[g][e] - m) * 1.4426950408889634f))
          B2_FU_IN(a[e] += X[g][e])
          const float s = fuse_group_reduce((a[0] + a[1]) + (a[2] + a[3]), add_f, slot, T, gi, gl, turn);
          const float rs = rcp_nr(s);
          B2_FU_ALL(X[g][e] *= rs)
          break;
        }
#define B2_FU_INT(CODE, EXPR) \
        case CODE: B2_FU_ALL(const uint32_t x = __float_as_uint(X[g][e]), y = __float_as_uint(Y[g][e]); (void)y; X[g][e] = __uint_as_float(EXPR)) break;
        B2_FU_INT(kFuIAdd, x + y)
        B2_FU_INT(kFuISub, x - y)
        B2_FU_INT(kFuIRSub, y - x)
        B2_FU_INT(kFuIMul, x * y)
        B2_FU_INT(kFuIAnd, x & y)
        B2_FU_INT(kFuIOr, x | y)
        B2_FU_INT(kFuIXor, x ^ y)
        B2_FU_INT(kFuIMax, static_cast<uint32_t>(max(static_cast<int32_t>(x), static_cast<int32_t>(y))))
        B2_FU_INT(kFuIMin, static_cast<uint32_t>(min(static_cast<int32_t>(x), static_cast<int32_t>(y))))
        B2_FU_INT(kFuUMax, max(x, y))
        B2_FU_INT(kFuUMin, min(x, y))
        B2_FU_INT(kFuINot, ~x)
        B2_FU_INT(kFuINeg, 0u - x)
#undef B2_FU_INT
        case kFuCarrySum: {
          float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          B2_FU_IN(a[e] += X[g][e])
          csum += (a[0] + a[1]) + (a[2] + a[3]);
          break;
        }
        case kFuCarrySumSq: {
          float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          B2_FU_IN(a[e] = __fadd_rn(a[e], __fmul_rn(X[g][e], X[g][e])))
          csum += (a[0] + a[1]) + (a[2] + a[3]);
          break;
        }
        default: break;
      }
    }
    buf ^= 1u;
#undef B2_FU_IN
#undef B2_FU_ALL
  }
  cp_async_wait_all();
  return csum;
}

static __device__ __noinline__ void row_pipe_tiles(const Lane &L, const DTask &t, const DFuse &f, uint32_t tile_lo, uint32_t tile_hi);

static __device__ __noinline__ void flat_pipe_tiles(const Lane &L, const DFuse &f, uint32_t tile_lo, uint32_t tile_hi);

static __device__ __noinline__ void fuse_rows_tiles(const Lane &L, const DTask &t, uint32_t tile_lo, uint32_t tile_hi) {
  const KParams &P = *L.P;
  const DFuse &f = *reinterpret_cast<const DFuse *>(planned_desc(L, t));
  if (f.flat) { flat_pipe_tiles(L, f, tile_lo, tile_hi); return; }
  if (f.pipe.flags) { row_pipe_tiles(L, t, f, tile_lo, tile_hi); return; }
  const DFuStep *ws = reinterpret_cast<const DFuStep *>(&f + 1);
  const uint32_t cols = f.cols, hi = min(tile_hi, f.rows), n = f.n_steps;
  FuStep *steps = reinterpret_cast<FuStep *>(L.smem + kFuseSteps);
  uint32_t *loads = reinterpret_cast<uint32_t *>(L.smem + kSmemChain);
  // Threads per row: 4 groups of 4 elements per thread (8, of which X and Y alone take 64 registers, only for rows past
  // 8192 elements); as many rows in flight as that allows, unless the lane has fewer rows than groups - then more threads
  // share a row.
  uint32_t T = 32u;
  while (T < 512u && (cols > T * 16u || (hi - tile_lo) * T * 2u <= L.nthr)) T *= 2u;
  const uint32_t per = (cols + 4u * T - 1u) / (4u * T);
  const uint32_t G = per <= 1u ? 1u : per <= 2u ? 2u : per <= 4u ? 4u : 8u;
  if (L.tid < n) {
    const DFuStep w = ws[L.tid];
    FuStep &d = steps[L.tid];
    d.code = w.code; d.dt = w.dt; d.s = w.s; d.t = w.t; d.reg = w.reg; d.slot = kFuNoSlot;
    d.ptr = w.ptr ? resolve(P, w.ptr) : nullptr;
  }
  __syncthreads();
  // staging room: column vectors first, then two buffers per dense load while they fit (every thread walks the list and
  // decides alike)
  bool rare = false;
  for (uint32_t i = 0; i < n; ++i) {
    const uint32_t k = ws[i].code;
    rare = rare || k == kFuDiv || k == kFuRDiv || k == kFuDivS || k == kFuExp || k == kFuTanh || k == kFuSqrt || k == kFuRsqrt || k == kFuLog;
  }
  uint32_t used = kFuseData, slots = 0, n_loads = 0;
  const uint32_t per_slot = 2u * G * L.nthr * 16u;
  for (uint32_t i = 0; i < n; ++i) {
    const uint32_t code = ws[i].code;
    if (code != kFuRowVecY) continue;
    const uint32_t bytes = cols * dt_size(ws[i].dt), b = (bytes + 15u) & ~15u;
    if (hi - tile_lo <= 1u || used + b + per_slot > L.smem_bytes) continue;
    const uint8_t *src = steps[i].ptr;
    const uint32_t words = bytes / 4u;
    for (uint32_t k = L.tid; k < words; k += L.nthr) reinterpret_cast<uint32_t *>(L.smem + used)[k] = ldg_u32(src + 4u * k);
    if (L.tid == 0) {
      if (bytes % 4u) *reinterpret_cast<uint16_t *>(L.smem + used + 4u * words) = static_cast<uint16_t>(ldg_u16(src + 4u * words));
      steps[i].slot = used;
    }
    used += b;
  }
  used = (used + 127u) & ~127u;
  const uint32_t fit = f.vec && used < L.smem_bytes ? (L.smem_bytes - used) / per_slot : 0u;
  for (uint32_t i = 0; i < n; ++i) {
    if (ws[i].code > kFuLoadY) continue;
    if (L.tid == 0) {
      loads[n_loads] = i;
      if (slots < fit) steps[i].slot = slots;
    }
    if (slots < fit) ++slots;
    ++n_loads;
  }
  __syncthreads();
  float csum = 0.0f;
  if (tile_lo < hi) {
#define B2_FU_RUN2(GG, RR)                                                                                                 \
  (f.vec ? fuse_rows_run<GG, true, RR>(L.tid, L.nthr, T, tile_lo, hi, cols, n, used, slots, n_loads, f.n_elems)            \
         : fuse_rows_run<GG, false, RR>(L.tid, L.nthr, T, tile_lo, hi, cols, n, used, 0u, n_loads, f.n_elems))
#define B2_FU_RUN(GG) case GG: csum = rare ? B2_FU_RUN2(GG, true) : B2_FU_RUN2(GG, false); break;
    switch (G) { B2_FU_RUN(1) B2_FU_RUN(2) B2_FU_RUN(4) default: B2_FU_RUN(8) }
#undef B2_FU_RUN
#undef B2_FU_RUN2
  }
  if (f.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(P, f.total)), t.p[3], f.n_owner_lanes);
}

}  // namespace b2

#include "ops_flatpipe.cuh"
#include "ops_rowpipe.cuh"
#endif
