// Products on the CUDA cores for re-planned programs (kTopSgemm): f32 operands, and 16-bit ones whose layout the tensor
// cores cannot be fed; f32 accumulation with FMA; the store epilogue of ops_gemm.cuh's kinds.
//
// Bound: FFMA issue (36 T FMA/s on 148 SMs) for large products, latency for small ones. The wire op's 128 x 128 tiles gave
// config 1 (256 x 64) two lanes and one scalar load per element behind a dtype switch: 62 us.
//
// Tiles from 128 x 64 down to 16 x 16 so that small products reach most lanes; what threads a tile does not need split K:
// KS slices of the CTA take every KS-th block of 16 k, each with its own ring of shared-memory blocks and its own named
// barrier, and their sums meet in shared memory in slice order. f32 operands come by cp.async, three blocks ahead (16 bytes
// where the rows are the unit-stride axis, else 4 and transposed on the way); 16-bit ones pass through registers, one block
// ahead. Operands are addressed as base + row part + k part (any view that separates there).
#ifndef B2VM_OPS_SGEMM_CUH_
#define B2VM_OPS_SGEMM_CUH_

#include "dev_common.cuh"
#include "ops_ew.cuh"
#include "ops_fuse.cuh"
#include "plan_format.h"

namespace b2 {

constexpr int kSgBK = 16;
constexpr uint32_t kSgTabA = kSmemSys, kSgTabB = kSgTabA + 512u, kSgData = kSgTabB + 512u;   // row parts of the tile's rows / columns, then data
template <int V> struct SgInt { static constexpr int value = V; };

// Offset of element (row, 0) / (0, k) in elements.
__device__ __forceinline__ uint32_t sg_row(const DSgOperand &o, uint32_t r) {
  if (!o.viewed) return o.off + r * o.rs;
  return static_cast<uint32_t>(view_index(o.v, o.row_major ? r * o.inner : r));
}
__device__ __forceinline__ uint32_t sg_k(const DSgOperand &o, uint32_t k) {
  if (!o.viewed) return k * o.ks;
  return static_cast<uint32_t>(view_index(o.v, o.row_major ? k : k * o.inner) - o.v.off);
}
__device__ __forceinline__ float sg_epilogue(const DSgemm &g, const uint8_t *res, float v, uint32_t r, uint32_t c, float &csum) {
  const uint32_t fl = g.epi;
  if (fl & kGeQuant0) v = quantize(v, g.qdt);
  if (fl & kGeGelu) v = gelu_tanh(v);
  if (fl & kGeScale0) v = __fmul_rn(v, g.s0);
  if (fl & kGeMaxS) v = np_max(v, g.s1);
  if (fl & kGeRes) {
    const float y = loadf(res, g.rdt, static_cast<int64_t>(r) * g.N + c);
    switch (fl & kGeResMask) {
      case kGeResAdd: v = __fadd_rn(v, y); break;
      case kGeResSub: v = __fsub_rn(v, y); break;
      case kGeResRSub: v = __fsub_rn(y, v); break;
      case kGeResMul: v = __fmul_rn(v, y); break;
      default: v = __fmul_rn(v, gelu_grad(y, g.gg)); break;
    }
  }
  if (fl & kGeCarrySq) csum = __fadd_rn(csum, __fmul_rn(v, v));
  if (fl & kGeScale1) v = __fmul_rn(v, g.s1);
  return v;
}

// N consecutive floats of shared memory.
template <int N>
__device__ __forceinline__ void sg_lds(const float *p, float (&x)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      const float4 f = reinterpret_cast<const float4 *>(p)[i];
      x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
    }
  } else {
    static_assert(N == 2, "pairs or fours");
    const float2 f = *reinterpret_cast<const float2 *>(p);
    x[0] = f.x; x[1] = f.y;
  }
}

// One block of an f32 operand (T rows of A, or columns of B, x 16 k) on its way to shared memory, k-major with pitch T + 4; what
// lies outside is zero. TH threads, `st` this one.
template <int T, int TH>
__device__ __forceinline__ void sg_copy(uint32_t dst, const uint8_t *p, const DSgOperand &o, const uint32_t *tab, uint32_t st, uint32_t first, uint32_t limit,
                                        uint32_t k0, uint32_t K) {
  constexpr int PITCH = T + 4;
  if (o.mode == kSgVecR) {
#pragma unroll
    for (int q = 0; q < T * kSgBK / 4 / TH; ++q) {
      const uint32_t w = st + q * TH, row = 4u * (w % (T / 4)), kk = w / (T / 4), k = k0 + kk;
      const bool in = first + row < limit && k < K;
      cp_async_16_zfill(dst + (kk * PITCH + row) * 4u, p + (static_cast<size_t>(tab[row]) + static_cast<size_t>(in ? k : 0u) * o.ks) * 4u, in ? 16u : 0u);
    }
  } else if (o.k_fast) {
#pragma unroll
    for (int q = 0; q < T * kSgBK / TH; ++q) {
      const uint32_t w = st + q * TH, row = w / kSgBK, kk = w % kSgBK, k = k0 + kk;
      const bool in = k < K;
      cp_async_4_zfill(dst + (kk * PITCH + row) * 4u, p + (static_cast<size_t>(tab[row]) + sg_k(o, in ? k : 0u)) * 4u, in ? 4u : 0u);
    }
  } else {
#pragma unroll
    for (int q = 0; q < T * kSgBK / TH; ++q) {
      const uint32_t w = st + q * TH, row = w % T, kk = w / T, k = k0 + kk;
      const bool in = k < K;
      cp_async_4_zfill(dst + (kk * PITCH + row) * 4u, p + (static_cast<size_t>(tab[row]) + sg_k(o, in ? k : 0u)) * 4u, in ? 4u : 0u);
    }
  }
}
// One block of a 16-bit operand into registers ...
template <int T, int TH>
__device__ __forceinline__ void sg_fetch(uint32_t (&v)[T * kSgBK / TH], const uint8_t *p, const DSgOperand &o, const uint32_t *tab, uint32_t st, uint32_t k0, uint32_t K) {
#pragma unroll
  for (int q = 0; q < T * kSgBK / TH; ++q) {
    const uint32_t w = st + q * TH;
    const uint32_t row = o.k_fast ? w / kSgBK : w % T, k = min(k0 + (o.k_fast ? w % kSgBK : w / T), K - 1u);
    v[q] = reinterpret_cast<const uint16_t *>(p)[static_cast<size_t>(tab[row]) + sg_k(o, k)];
  }
}
// ... and from there, as f32, to shared memory.
template <int T, int TH>
__device__ __forceinline__ void sg_put(const uint32_t (&v)[T * kSgBK / TH], float *d, uint32_t dt, const DSgOperand &o, uint32_t st, uint32_t k0, uint32_t K) {
#pragma unroll
  for (int q = 0; q < T * kSgBK / TH; ++q) {
    const uint32_t w = st + q * TH, row = o.k_fast ? w / kSgBK : w % T, kk = o.k_fast ? w % kSgBK : w / T;
    const float f = dt == kBF16 ? __uint_as_float(v[q] << 16) : f16_bits_to_f32(v[q]);
    d[kk * (T + 4) + row] = k0 + kk < K ? f : 0.0f;
  }
}

// A lane's tiles of TM x TN. MM x NN outputs per thread of a slice.
template <bool F32, int TM, int TN, int MM, int NN>
static __device__ __noinline__ void sgemm_run(const Lane &L, const DSgemm &g, uint32_t slot, uint32_t n_slots, float &csum) {
  constexpr int TR = TM / MM, TC = TN / NN, TH = TR * TC, KS = 512 / TH;       // threads of a slice; slices
  constexpr int PA = TM + 4, PB = TN + 4;                                      // pitches (16-byte rows, spread over banks)
  constexpr int BUF = kSgBK * (PA + PB), ST = F32 ? 4 : 2;
  static_assert(TH % 32 == 0 && MM % 2 == 0, "whole warps, pairs of rows");
  static_assert(kSgData + (ST * BUF * KS > KS * TM * TN ? ST * BUF * KS : KS * TM * TN) * 4 <= 216 * 1024, "fits the lane's shared memory");
  const KParams &P = *L.P;
  uint32_t *ra = reinterpret_cast<uint32_t *>(L.smem + kSgTabA), *rb = reinterpret_cast<uint32_t *>(L.smem + kSgTabB);
  float *data = reinterpret_cast<float *>(L.smem + kSgData);
  const uint8_t *A = resolve(P, g.a.ptr), *B = resolve(P, g.b.ptr);
  const uint8_t *res = (g.epi & kGeRes) ? resolve(P, g.res) : nullptr;
  uint8_t *out0 = g.out0 ? resolve(P, g.out0) : nullptr, *out1 = g.out1 ? resolve(P, g.out1) : nullptr;
  const uint32_t M = g.M, N = g.N, K = g.K;
  const uint32_t sl = L.tid / TH, st = L.tid % TH, tr = st / TC, tc = st % TC;
  float *buf0 = data + sl * ST * BUF;
  const uint32_t sbuf = smem_addr(buf0);
  const uint32_t tn = (N + TN - 1u) / TN, tiles = ((M + TM - 1u) / TM) * tn;
  const uint32_t nkb = (K + kSgBK - 1u) / kSgBK, mine = nkb > sl ? (nkb - sl + KS - 1u) / KS : 0u;   // this slice's blocks
  for (uint32_t tile = slot; tile < tiles; tile += n_slots) {
    const uint32_t r0 = (tile / tn) * TM, c0 = (tile % tn) * TN;
    __syncthreads();
    for (uint32_t i = L.tid; i < TM; i += 512u) ra[i] = sg_row(g.a, min(r0 + i, M - 1u));
    for (uint32_t i = L.tid; i < TN; i += 512u) rb[i] = sg_row(g.b, min(c0 + i, N - 1u));
    __syncthreads();
    unsigned long long acc[MM / 2][NN];        // f32 pairs: two rows of a column
#pragma unroll
    for (int i = 0; i < MM / 2; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) acc[i][j] = 0ull;
    auto block = [&](uint32_t i) {
      const float *as = buf0 + (i % ST) * BUF + tr * MM, *bs = buf0 + (i % ST) * BUF + kSgBK * PA + tc * NN;
#pragma unroll
      for (int k = 0; k < kSgBK; ++k) {
        float x[MM], y[NN];
        sg_lds<MM>(as + k * PA, x);
        sg_lds<NN>(bs + k * PB, y);
#pragma unroll
        for (int j = 0; j < NN; ++j) {
          const unsigned long long yy = pack_f32x2(y[j], y[j]);
#pragma unroll
          for (int r = 0; r < MM / 2; ++r) acc[r][j] = fma_f32x2(pack_f32x2(x[2 * r], x[2 * r + 1]), yy, acc[r][j]);
        }
      }
    };
    if constexpr (F32) {
      auto copy = [&](uint32_t i) {
        const uint32_t k0 = (sl + i * KS) * kSgBK, d = sbuf + (i % ST) * BUF * 4u;
        if (i < mine) {
          sg_copy<TM, TH>(d, A, g.a, ra, st, r0, M, k0, K);
          sg_copy<TN, TH>(d + kSgBK * PA * 4u, B, g.b, rb, st, c0, N, k0, K);
        }
        cp_async_commit();
      };
      for (uint32_t i = 0; i < ST - 1; ++i) copy(i);
#pragma unroll 1
      for (uint32_t i = 0; i < mine; ++i) {
        cp_async_wait<ST - 2>();
        bar_sync(1 + static_cast<int>(sl), TH);           // block i is there, and everyone is done with the one before it
        copy(i + ST - 1);
        block(i);
      }
      cp_async_wait_all();
    } else {
      uint32_t va[TM * kSgBK / TH], vb[TN * kSgBK / TH];
      auto fetch = [&](uint32_t i) {
        sg_fetch<TM, TH>(va, A, g.a, ra, st, (sl + i * KS) * kSgBK, K);
        sg_fetch<TN, TH>(vb, B, g.b, rb, st, (sl + i * KS) * kSgBK, K);
      };
      if (mine) fetch(0);
#pragma unroll 1
      for (uint32_t i = 0; i < mine; ++i) {
        float *as = buf0 + (i % ST) * BUF;
        sg_put<TM, TH>(va, as, g.adt, g.a, st, (sl + i * KS) * kSgBK, K);
        sg_put<TN, TH>(vb, as + kSgBK * PA, g.adt, g.b, st, (sl + i * KS) * kSgBK, K);
        bar_sync(1 + static_cast<int>(sl), TH);
        if (i + 1u < mine) fetch(i + 1u);
        block(i);
      }
    }
    // the slices' sums, in slice order
    __syncthreads();
    float *part = data + sl * (TM * TN);
#pragma unroll
    for (int i = 0; i < MM / 2; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) {
        float *d = part + (tr * MM + 2 * i) * TN + tc * NN + j;
        unpack_f32x2(acc[i][j], d[0], d[TN]);
      }
    __syncthreads();
    for (uint32_t e = L.tid; e < TM * TN; e += 512u) {
      const uint32_t r = r0 + e / TN, c = c0 + e % TN;
      if (r >= M || c >= N) continue;
      float v = data[e];
#pragma unroll
      for (int s = 1; s < KS; ++s) v += data[s * (TM * TN) + e];
      if (out0) storef(out0, g.dt0, static_cast<int64_t>(r) * N + c, v);
      v = sg_epilogue(g, res, v, r, c, csum);
      if (out1) storef(out1, g.dt1, static_cast<int64_t>(r) * N + c, v);
    }
  }
}

template <bool F32>
__device__ __forceinline__ void sgemm_shape(const Lane &L, const DSgemm &g, uint32_t slot, uint32_t n_slots, float &csum) {
  switch (g.shape) {
    case 0: sgemm_run<F32, 128, 64, 8, 4>(L, g, slot, n_slots, csum); break;
    case 1: sgemm_run<F32, 64, 64, 4, 4>(L, g, slot, n_slots, csum); break;
    case 2: sgemm_run<F32, 64, 32, 4, 4>(L, g, slot, n_slots, csum); break;
    case 3: sgemm_run<F32, 32, 32, 4, 4>(L, g, slot, n_slots, csum); break;
    default: sgemm_run<F32, 16, 16, 2, 2>(L, g, slot, n_slots, csum); break;
  }
}
static __device__ __noinline__ void sgemm_tiles(const Lane &L, const DTask &t, uint32_t slot, uint32_t n_slots) {
  const DSgemm &g = *reinterpret_cast<const DSgemm *>(planned_desc(L, t));
  float csum = 0.0f;
  if (g.adt == kF32) sgemm_shape<true>(L, g, slot, n_slots, csum);
  else sgemm_shape<false>(L, g, slot, n_slots, csum);
  if (g.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(*L.P, g.total)), t.p[3], g.n_owner_lanes);
}

}  // namespace b2
#endif
