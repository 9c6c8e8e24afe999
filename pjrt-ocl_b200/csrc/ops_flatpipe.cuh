// Flat elementwise chains of 4-byte elements with one to three binary ops, X = load; X = X op load, ...; store, as
// straight-line code (kTopFuseRows with DFuse::flat set): what config 2's integer chain is. A thread owns two groups of 4
// consecutive elements of a piece (up to 4096 elements; fewer where the whole list would not reach every lane); all operands of the next piece are under way as asynchronous copies
// into the thread's own staging words while the current one is worked on (64 KB per SM in flight with four operands).
// Bound: HBM. i32 max((a + b) ^ c, d), 8192 x 4096: 141 us as an interpreted chain, 115 us so (5.8 TB/s);
// 1135 x 128 14.1 -> 10.0 us (one piece a lane).
#ifndef B2VM_OPS_FLATPIPE_CUH_
#define B2VM_OPS_FLATPIPE_CUH_

#include "ops_fuse.cuh"

namespace b2 {

__device__ __forceinline__ void flat_op(uint32_t code, uint32_t (&x)[8], const uint32_t (&y)[8]) {
#define B2_FLAT_I(C, EXPR) case C: _Pragma("unroll") for (int i = 0; i < 8; ++i) { const uint32_t a = x[i], b = y[i]; x[i] = (EXPR); } break;
#define B2_FLAT_F(C, EXPR) \
  case C: _Pragma("unroll") for (int i = 0; i < 8; ++i) { const float a = __uint_as_float(x[i]), b = __uint_as_float(y[i]); x[i] = __float_as_uint(EXPR); } break;
  switch (code) {
    B2_FLAT_I(kFuIAdd, a + b)
    B2_FLAT_I(kFuISub, a - b)
    B2_FLAT_I(kFuIRSub, b - a)
    B2_FLAT_I(kFuIMul, a * b)
    B2_FLAT_I(kFuIAnd, a & b)
    B2_FLAT_I(kFuIOr, a | b)
    B2_FLAT_I(kFuIXor, a ^ b)
    B2_FLAT_I(kFuIMax, static_cast<uint32_t>(max(static_cast<int32_t>(a), static_cast<int32_t>(b))))
    B2_FLAT_I(kFuIMin, static_cast<uint32_t>(min(static_cast<int32_t>(a), static_cast<int32_t>(b))))
    B2_FLAT_I(kFuUMax, max(a, b))
    B2_FLAT_I(kFuUMin, min(a, b))
    B2_FLAT_F(kFuAdd, __fadd_rn(a, b))
    B2_FLAT_F(kFuMul, __fmul_rn(a, b))
    B2_FLAT_F(kFuSub, __fsub_rn(a, b))
    B2_FLAT_F(kFuRSub, __fsub_rn(b, a))
    B2_FLAT_F(kFuMax, np_max(a, b))
    B2_FLAT_F(kFuMin, np_min(a, b))
    default: break;
  }
#undef B2_FLAT_F
#undef B2_FLAT_I
}

template <int NB>      // binary ops
static __device__ __noinline__ void flat_run(const Lane &L, const DFuse &f, uint32_t lo, uint32_t hi) {
  const KParams &P = *L.P;
  const DFuStep *st = reinterpret_cast<const DFuStep *>(&f + 1);
  const uint8_t *src[NB + 1];
  uint32_t code[NB];
  src[0] = resolve(P, st[0].ptr);
#pragma unroll
  for (int k = 0; k < NB; ++k) { src[k + 1] = resolve(P, st[1 + 2 * k].ptr); code[k] = st[2 + 2 * k].code; }
  uint8_t *dst = resolve(P, st[1 + 2 * NB].ptr);
  const uint32_t sb = smem_addr(L.smem + kFuseData) + L.tid * 16u;
  constexpr uint32_t kGroup = 512u * 16u, kBuf = (NB + 1) * 2u * kGroup;
  const uint32_t piece_n = f.cols;         // <= 4096: 512 threads x 2 groups x 4 elements
  const uint32_t n0 = L.tid * 4u < piece_n ? f.n_elems : 0u, n1 = L.tid * 4u + 2048u < piece_n ? f.n_elems : 0u;      // where this thread's groups end
  auto start = [&](uint32_t piece, uint32_t buf) {
    const uint32_t e0 = piece * piece_n + L.tid * 4u;
#pragma unroll
    for (int k = 0; k <= NB; ++k)
#pragma unroll
      for (uint32_t g = 0; g < 2u; ++g) {
        const uint32_t e = e0 + g * 2048u;
        if (e < (g ? n1 : n0)) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sb + buf * kBuf + (k * 2u + g) * kGroup), "l"(src[k] + static_cast<size_t>(e) * 4u) : "memory");
      }
    cp_async_commit();
  };
  start(lo, 0u);
  uint32_t buf = 0;
  for (uint32_t piece = lo; piece < hi; ++piece) {
    cp_async_wait<0>();
    if (piece + 1u < hi) start(piece + 1u, buf ^ 1u);
    const uint8_t *s = L.smem + kFuseData + L.tid * 16u + buf * kBuf;
    uint32_t x[8], y[8];
    auto take = [&](uint32_t (&r)[8], int k) {
      const uint4 a = *reinterpret_cast<const uint4 *>(s + (k * 2) * kGroup), b = *reinterpret_cast<const uint4 *>(s + (k * 2 + 1) * kGroup);
      r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w; r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    };
    take(x, 0);
#pragma unroll
    for (int k = 0; k < NB; ++k) { take(y, k + 1); flat_op(code[k], x, y); }
    const uint32_t e = piece * piece_n + L.tid * 4u;
    if (e < n0) stg_v4(dst + static_cast<size_t>(e) * 4u, make_uint4(x[0], x[1], x[2], x[3]));
    if (e + 2048u < n1) stg_v4(dst + static_cast<size_t>(e + 2048u) * 4u, make_uint4(x[4], x[5], x[6], x[7]));
    buf ^= 1u;
  }
  cp_async_wait_all();
}

static __device__ __noinline__ void flat_pipe_tiles(const Lane &L, const DFuse &f, uint32_t tile_lo, uint32_t tile_hi) {
  const uint32_t hi = min(tile_hi, f.rows);
  if (tile_lo >= hi) return;
  switch (f.flat) {
    case 1: flat_run<1>(L, f, tile_lo, hi); break;
    case 2: flat_run<2>(L, f, tile_lo, hi); break;
    default: flat_run<3>(L, f, tile_lo, hi); break;
  }
}

}  // namespace b2
#endif
