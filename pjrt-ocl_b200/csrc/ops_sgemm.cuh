// Products on the CUDA cores for re-planned programs (kTopSgemm): f32 operands, and 16-bit ones whose layout the tensor
// cores cannot be fed; f32 accumulation with FMA; the store epilogue of ops_gemm.cuh's kinds.
//
// Bound: FFMA issue (36 T FMA/s on 148 SMs) for large products, latency for small ones. The wire op's 128 x 128 tiles gave
// config 1 (256 x 64) two lanes and one scalar load per element behind a dtype switch: 62 us, 5 now; 1024 cubed 72 us (40 % of issue).
//
// Tiles from 128 x 64 down to 16 x 16 so that small products reach most lanes; what threads a tile does not need split K:
// KS slices of the CTA take every KS-th block of 16 k, each with its own ring of shared-memory blocks and its own named
// barrier, and their sums meet in shared memory in slice order. f32 operands come by cp.async, three blocks ahead (16 bytes
// where the rows are the unit-stride axis, else 4 and transposed on the way); 16-bit ones pass through registers, one block
// ahead.
#ifndef B2VM_OPS_SGEMM_CUH_
#define B2VM_OPS_SGEMM_CUH_

#include "dev_common.cuh"
#include "ops_ew.cuh"
#include "ops_fuse.cuh"
#include "plan_format.h"

namespace b2 {

constexpr int kSgBK = 16;
constexpr uint32_t kSgTab = kSmemSys, kSgData = kSgTab + 1024u;     // row parts of viewed operands (A 128, B 64), then data

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

// A thread's N of T rows (or columns) of a block: fours at 4 `t` and, for eight, at T / 2 + 4 `t`, so that a warp's threads (4 row
// groups x 8 column groups) read whole 64- and 128-byte pieces of shared memory.
template <int N, int T>
__device__ __forceinline__ uint32_t sg_at(uint32_t t, int i) {
  if constexpr (N == 8) return (i >> 2) * (T / 2) + 4u * t + (i & 3);
  else return N * t + i;
}
template <int N, int T>
__device__ __forceinline__ void sg_lds(const float *p, uint32_t t, float (&x)[N]) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 f = *reinterpret_cast<const float4 *>(p + sg_at<N, T>(t, i));
      x[i] = f.x; x[i + 1] = f.y; x[i + 2] = f.z; x[i + 3] = f.w;
    }
  } else {
    static_assert(N == 2, "pairs or fours");
    const float2 f = *reinterpret_cast<const float2 *>(p + 2u * t);
    x[0] = f.x; x[1] = f.y;
  }
}

// What a thread copies of an operand's block of T rows (or columns) x 16 k: elements (or fours of them along the rows) q = 0, 1, ...
// Either its row or its k stays. Worked out anew for every block: the accumulators leave no registers to keep it in.
template <int T, int TH>
struct SgThread {
  static constexpr int E = T * kSgBK / TH;     // elements
  uint32_t row, k, rq, kq;                     // of q = 0; per q
  bool four;
  __device__ __forceinline__ SgThread(const DSgOperand &o, uint32_t st) {
    static_assert(T <= TH && E <= 32, "one row, or one k, per thread");
    four = o.mode == kSgVecR;
    const bool kf = !four && o.k_fast != 0u;
    row = four ? 4u * (st % (T / 4)) : kf ? st / kSgBK : st % T;
    k = four ? st / (T / 4) : kf ? st % kSgBK : st / T;
    kq = four ? 4u * TH / T : kf ? 0u : TH / T;
    rq = kf ? TH / kSgBK : 0u;
  }
  __device__ __forceinline__ uint32_t start(const DSgOperand &o, uint32_t first, uint32_t k0) const { return o.off + (first + row) * o.rs + (k0 + k) * o.ks; }
  __device__ __forceinline__ uint32_t step(const DSgOperand &o) const { return rq * o.rs + kq * o.ks; }
  __device__ __forceinline__ uint32_t dst() const { return k * (T + 4) + row; }
  __device__ __forceinline__ uint32_t sstep() const { return kq * (T + 4) + rq; }
  __device__ __forceinline__ bool in(int q, uint32_t first, uint32_t limit, uint32_t k0, uint32_t K) const {
    return first + row + q * rq < limit && k0 + k + q * kq < K;
  }
};
// Viewed operands: a row's part, a k's part.
__device__ __forceinline__ uint32_t sg_row(const DSgOperand &o, uint32_t r) { return static_cast<uint32_t>(view_index(o.v, o.row_major ? r * o.inner : r)); }
__device__ __forceinline__ uint32_t sg_k(const DSgOperand &o, uint32_t k) { return static_cast<uint32_t>(view_index(o.v, o.row_major ? k : k * o.inner) - o.v.off); }
// f32: the block from k0 to shared memory at `d`, k-major with pitch T + 4; what lies outside is zero.
template <int T, int TH>
__device__ __forceinline__ void sg_copy(uint32_t d, const uint8_t *base, const DSgOperand &o, const uint32_t *tab, uint32_t st, uint32_t first, uint32_t limit, uint32_t k0,
                                        uint32_t K) {
  const SgThread<T, TH> t(o, st);
  const uint32_t ds = t.sstep() * 4u;
  if (o.viewed) {
    d += t.dst() * 4u;
    uint32_t kp = sg_k(o, min(k0 + t.k, K - 1u));
#pragma unroll 4
    for (uint32_t q = 0; q < static_cast<uint32_t>(SgThread<T, TH>::E); ++q, d += ds) {
      const bool in = t.in(q, first, limit, k0, K);
      if (t.kq && in) kp = sg_k(o, k0 + t.k + q * t.kq);
      cp_async_4_zfill(d, in ? base + (static_cast<size_t>(tab[t.row + q * t.rq]) + kp) * 4u : base, in ? 4u : 0u);
    }
    return;
  }
  const size_t step = static_cast<size_t>(t.step(o)) * 4u;
  const uint8_t *s = base + static_cast<size_t>(t.start(o, first, k0)) * 4u;
  d += t.dst() * 4u;
  const bool whole = first + T <= limit && k0 + kSgBK <= K;
  if (whole && t.four) {
#pragma unroll
    for (int q = 0; q < SgThread<T, TH>::E / 4; ++q, s += step, d += ds) cp_async_16_zfill(d, s, 16u);
  } else if (whole) {
#pragma unroll
    for (int q = 0; q < SgThread<T, TH>::E; ++q, s += step, d += ds) cp_async_4_zfill(d, s, 4u);
  } else {
    // an address outside the buffer is not even named
    const uint32_t n = t.four ? SgThread<T, TH>::E / 4 : SgThread<T, TH>::E;
#pragma unroll 1
    for (uint32_t q = 0; q < n; ++q, s += step, d += ds) {
      const bool in = t.in(q, first, limit, k0, K);
      if (t.four) cp_async_16_zfill(d, in ? s : base, in ? 16u : 0u);
      else cp_async_4_zfill(d, in ? s : base, in ? 4u : 0u);
    }
  }
}
// 16-bit: the block into registers ...
template <int T, int TH>
__device__ __forceinline__ void sg_fetch(uint32_t (&v)[SgThread<T, TH>::E], const uint8_t *base, const DSgOperand &o, const uint32_t *tab, uint32_t st, uint32_t first,
                                         uint32_t limit, uint32_t k0, uint32_t K) {
  const SgThread<T, TH> t(o, st);
  if (o.viewed) {
#pragma unroll
    for (int q = 0; q < SgThread<T, TH>::E; ++q)
      v[q] = t.in(q, first, limit, k0, K) ? reinterpret_cast<const uint16_t *>(base)[static_cast<size_t>(tab[t.row + q * t.rq]) + sg_k(o, k0 + t.k + q * t.kq)] : 0u;
    return;
  }
  const size_t step = static_cast<size_t>(t.step(o)) * 2u;
  const uint8_t *s = base + static_cast<size_t>(t.start(o, first, k0)) * 2u;
#pragma unroll
  for (int q = 0; q < SgThread<T, TH>::E; ++q, s += step) v[q] = t.in(q, first, limit, k0, K) ? *reinterpret_cast<const uint16_t *>(s) : 0u;
}
// ... and from there, as f32, to shared memory.
template <int T, int TH>
__device__ __forceinline__ void sg_put(const uint32_t (&v)[SgThread<T, TH>::E], float *d, uint32_t dt, const DSgOperand &o, uint32_t st) {
  const SgThread<T, TH> t(o, st);
  const uint32_t ds = t.sstep();
  d += t.dst();
#pragma unroll
  for (int q = 0; q < SgThread<T, TH>::E; ++q, d += ds) *d = dt == kBF16 ? __uint_as_float(v[q] << 16) : f16_bits_to_f32(v[q]);
}

// A lane's tiles of TM x TN. MM x NN outputs per thread of a slice.
template <bool F32, int TM, int TN, int MM, int NN, int ST>
static __device__ __noinline__ void sgemm_run(const Lane &L, const DSgemm &g, uint32_t slot, uint32_t n_slots, float &csum) {
  constexpr int TR = TM / MM, TC = TN / NN, TH = TR * TC, KS = 512 / TH;       // threads of a slice; slices
  constexpr int PA = TM + 4, PB = TN + 4;                                      // pitches (16-byte rows, spread over banks)
  constexpr int BUF = kSgBK * (PA + PB);
  static_assert(TH % 32 == 0 && TC == 8 && MM % 2 == 0, "whole warps of 4 x 8 threads, pairs of rows");
  static_assert(kSgData + (ST * BUF * KS > KS * TM * TN ? ST * BUF * KS : KS * TM * TN) * 4 <= 216 * 1024, "fits the lane's shared memory");
  const KParams &P = *L.P;
  uint32_t *ra = reinterpret_cast<uint32_t *>(L.smem + kSgTab), *rb = ra + 128;
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
    if (g.a.viewed | g.b.viewed) {
      if (g.a.viewed) for (uint32_t i = L.tid; i < TM; i += 512u) ra[i] = sg_row(g.a, min(r0 + i, M - 1u));
      if (g.b.viewed) for (uint32_t i = L.tid; i < TN; i += 512u) rb[i] = sg_row(g.b, min(c0 + i, N - 1u));
      __syncthreads();
    }
    unsigned long long acc[MM / 2][NN];        // f32 pairs: two rows of a column
#pragma unroll
    for (int i = 0; i < MM / 2; ++i)
#pragma unroll
      for (int j = 0; j < NN; ++j) acc[i][j] = 0ull;
    auto block = [&](uint32_t i) {
      const float *as = buf0 + (i % ST) * BUF, *bs = as + kSgBK * PA;
#pragma unroll 4
      for (int k = 0; k < kSgBK; ++k) {
        float x[MM], y[NN];
        sg_lds<MM, TM>(as + k * PA, tr, x);
        sg_lds<NN, TN>(bs + k * PB, tc, y);
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
#pragma unroll 1
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
      uint32_t va[SgThread<TM, TH>::E], vb[SgThread<TN, TH>::E];
      auto fetch = [&](uint32_t i) {
        const uint32_t k0 = (sl + i * KS) * kSgBK;
        sg_fetch<TM, TH>(va, A, g.a, ra, st, r0, M, k0, K);
        sg_fetch<TN, TH>(vb, B, g.b, rb, st, c0, N, k0, K);
      };
      if (mine) fetch(0);
#pragma unroll 1
      for (uint32_t i = 0; i < mine; ++i) {
        float *as = buf0 + (i % ST) * BUF;
        sg_put<TM, TH>(va, as, g.adt, g.a, st);
        sg_put<TN, TH>(vb, as + kSgBK * PA, g.adt, g.b, st);
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
        float *d = part + sg_at<MM, TM>(tr, 2 * i) * TN + sg_at<NN, TN>(tc, j);
        unpack_f32x2(acc[i][j], d[0], d[TN]);
      }
    __syncthreads();
#pragma unroll 1
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
  constexpr int ST = F32 ? 4 : 2;
  switch (g.shape) {
    case 0: sgemm_run<F32, 128, 64, 8, 8, ST>(L, g, slot, n_slots, csum); break;
    case 1: sgemm_run<F32, 64, 64, 8, 8, F32 ? 3 : 2>(L, g, slot, n_slots, csum); break;
    case 2: sgemm_run<F32, 64, 32, 8, 4, F32 ? 3 : 2>(L, g, slot, n_slots, csum); break;
    case 3: sgemm_run<F32, 32, 32, 4, 4, ST>(L, g, slot, n_slots, csum); break;
    default: sgemm_run<F32, 16, 16, 2, 2, ST>(L, g, slot, n_slots, csum); break;
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
