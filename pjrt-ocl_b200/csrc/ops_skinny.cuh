// Products with at most 32 rows (a decode step) of re-planned programs (kTopSkinny): bf16 / f16 operands, f32
// accumulation, the store epilogue of ops_sgemm.cuh.
//
// Bound: reading the weights once; at these sizes that is latency. On 128-row tensor-core tiles such a product had N / 64
// lanes at work, each walking all of K alone (a phase of 32 x 1024 by 1024 x 4096: 20 us, now 11; 32 x 4096 by 4096 x 1024:
// 38 us, now 17; 1 x 512 by 512 x 512: 12-14 us, now 7).
// Here a tile is all rows by 8, 16 or 32 columns, so that every lane has its own piece of the weights, and the lane's 16 warps
// split K: warp w takes every 16th group of 32 k, through a ring of its own in shared memory (16-byte asynchronous copies,
// several groups ahead, no barrier among the warps), multiplies with mma.m16n8k16 (the tensor pipe is not what bounds it, and a tcgen05
// tile has 128 rows), and the warps' sums meet in shared memory in warp order.
// Rows that are an RMS norm's result are normed by every lane for itself, under the first weights' flight.
// A dynamic slice update that was all a product was for (a cache row) is its store's address.
// Ring block: A as rows of 64 bytes with their 16-byte pieces swizzled; B, columns contiguous: planes of 8 columns, 16 bytes per k;
// B, k contiguous: like A. ldmatrix reads each without bank conflicts.
#ifndef B2VM_OPS_SKINNY_CUH_
#define B2VM_OPS_SKINNY_CUH_

#include "ops_move.cuh"
#include "ops_sgemm.cuh"

namespace b2 {

constexpr uint32_t kSkWarps = 16, kSkRing = 12800;        // bytes of a warp's ring
constexpr uint32_t kSkNormRing = 8192, kSkNormRows = 65536;   // with the normed rows kept whole beside the rings: 32 rows x 1024

// The lane's copy of the normed rows: blocks of 32 k, each rows of 64 bytes like a ring block's. A warp takes every 16th row, 32 lanes
// x 8 elements at a time. Rows past M are zero.
static __device__ __noinline__ void skinny_norm(const Lane &L, const DSgemm &g, uint32_t rows) {
  const KParams &P = *L.P;
  const uint32_t w = L.tid / kWarp, l = L.tid % kWarp, K = g.K, dt = g.adt;
  const uint8_t *x = resolve(P, g.a.ptr), *gam = resolve(P, g.gamma);
  uint8_t *dst = L.smem + kSmemSys + kSkWarps * kSkNormRing;
#pragma unroll 1
  for (uint32_t r = w; r < rows; r += kSkWarps) {
    uint4 v[4];
    float ss = 0.0f, f[8];
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      const uint32_t k = 8u * (l + 32u * q);
      v[q] = r < g.M && k < K ? ldg_v4(x + (static_cast<size_t>(r) * K + k) * 2u) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      unpack8(v[q], dt, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss = fmaf(f[e], f[e], ss);
    }
    ss = warp_reduce(ss, [](float a, float b) { return a + b; });
    const float rs = rsqrtf(fmaf(ss, g.ns, g.nt));
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      const uint32_t p = l + 32u * q, k = 8u * p;
      if (k >= K) break;
      float y[8];
      uint32_t o[4];
      unpack8(v[q], dt, f);
      unpack8(ldg_v4(gam + k * 2u), dt, y);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float lo = __fmul_rn(__fmul_rn(f[2 * e], rs), y[2 * e]), hi = __fmul_rn(__fmul_rn(f[2 * e + 1], rs), y[2 * e + 1]);
        o[e] = dt == kBF16 ? cvt_bf16x2(hi, lo) : (f32_to_f16_bits(lo) | (f32_to_f16_bits(hi) << 16));
      }
      *reinterpret_cast<uint4 *>(dst + (p >> 2) * rows * 64u + r * 64u + (((p & 3u) ^ ((r >> 1) & 3u)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

template <int MT, int NB, bool NORM>
static __device__ __noinline__ void skinny_run(const Lane &L, const DSgemm &g, uint32_t slot, uint32_t n_slots, float &csum) {
  constexpr uint32_t kA = NORM ? 0u : 1024u * MT, kB = 512u * NB, kBlock = kA + kB, kRing = NORM ? kSkNormRing : kSkRing;
  constexpr uint32_t kDepth = kRing / kBlock > 8u ? 8u : kRing / kBlock;
  constexpr uint32_t ROWS = 16u * MT, COLS = 8u * NB;
  static_assert(kDepth >= 2u && ROWS * COLS * 4u <= kRing, "a block ahead; the sums fit over the rings");
  const KParams &P = *L.P;
  const uint8_t *A = resolve(P, g.a.ptr) + static_cast<size_t>(g.a.off) * 2u, *B = resolve(P, g.b.ptr) + static_cast<size_t>(g.b.off) * 2u;
  const uint8_t *res = (g.epi & kGeRes) ? resolve(P, g.res) : nullptr;
  uint8_t *out0 = g.out0 ? resolve(P, g.out0) : nullptr, *out1 = g.out1 ? resolve(P, g.out1) : nullptr;
  const uint32_t M = g.M, N = g.N, K = g.K, w = L.tid / kWarp, l = L.tid % kWarp;
  const size_t lda = static_cast<size_t>(g.a.rs) * 2u;
  const bool b_k = g.b.ks == 1u, bf = g.adt == kBF16;
  const size_t ldb = static_cast<size_t>(b_k ? g.b.rs : g.b.ks) * 2u;
  const uint32_t ring = smem_addr(L.smem + kSmemSys) + w * kRing, normed = smem_addr(L.smem + kSmemSys) + kSkWarps * kSkNormRing;
  float *part = reinterpret_cast<float *>(L.smem + kSmemSys);
  const uint32_t groups = (K + 31u) / 32u, mine = groups > w ? (groups - w + kSkWarps - 1u) / kSkWarps : 0u;
  const uint32_t tiles = (N + COLS - 1u) / COLS;
  bool first = true;
  const DMove *mv = g.move ? reinterpret_cast<const DMove *>(P.desc + g.move) : nullptr;
  for (uint32_t tile = slot; tile < tiles; tile += n_slots) {
    const uint32_t c0 = tile * COLS;
    __syncthreads();
    auto copy = [&](uint32_t i) {
      if (i < mine) {
        const uint32_t k0 = (w + i * kSkWarps) * 32u, d = ring + (i % kDepth) * kBlock;
        if constexpr (!NORM) {
#pragma unroll
          for (uint32_t q = 0; q < 2u * MT; ++q) {             // rows x four 16-byte pieces
            const uint32_t e = l + 32u * q, r = e >> 2, p = e & 3u, k = k0 + 8u * p;
            const bool in = r < M && k < K;
            cp_async_16_zfill(d + r * 64u + ((p ^ ((r >> 1) & 3u)) << 4), in ? A + r * lda + k * 2u : A, in ? 16u : 0u);
          }
        }
        if (b_k) {
#pragma unroll
          for (uint32_t q = 0; q < static_cast<uint32_t>(NB); ++q) {
            const uint32_t e = l + 32u * q, r = e >> 2, p = e & 3u, k = k0 + 8u * p;
            const bool in = c0 + r < N && k < K;
            cp_async_16_zfill(d + kA + r * 64u + ((p ^ ((r >> 1) & 3u)) << 4), in ? B + (c0 + r) * ldb + k * 2u : B, in ? 16u : 0u);
          }
        } else {
#pragma unroll
          for (uint32_t q = 0; q < static_cast<uint32_t>(NB); ++q) {
            const uint32_t e = l + 32u * q, kk = e / NB, nb = e % NB;
            const bool in = c0 + 8u * nb < N && k0 + kk < K;
            cp_async_16_zfill(d + kA + nb * 512u + kk * 16u, in ? B + (k0 + kk) * ldb + (c0 + 8u * nb) * 2u : B, in ? 16u : 0u);
          }
        }
      }
      cp_async_commit();
    };
    float acc[MT][NB][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.0f;
    // (not unrolled, here and below: a phase runs this code once, and fetching it is much of its time)
#pragma unroll 1
    for (uint32_t i = 0; i + 1u < kDepth; ++i) copy(i);
    const int64_t at = mv ? dyn_base(P, *mv) : 0;          // (its loads too under the weights' flight)
    if (NORM && first) {
      skinny_norm(L, g, ROWS);
      __syncthreads();
      first = false;
    }
#pragma unroll 1
    for (uint32_t i = 0; i < mine; ++i) {
      cp_async_wait<kDepth - 2>();
      __syncwarp();                        // the other threads' copies of block i, and their reads of the block before it
      copy(i + kDepth - 1u);
      const uint32_t d = ring + (i % kDepth) * kBlock, ad = NORM ? normed + (w + i * kSkWarps) * (ROWS * 64u) : d;
      uint32_t b[NB][4];
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        const uint32_t r = 8u * n + (l & 7u), p = l >> 3;
        if (b_k) ldmatrix_x4(b[n], d + kA + r * 64u + ((p ^ ((r >> 1) & 3u)) << 4));
        else ldmatrix_x4_trans(b[n], d + kA + n * 512u + l * 16u);
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
          const uint32_t r = 16u * m + (l & 15u), p = 2u * j + (l >> 4);
          uint32_t a[4];
          ldmatrix_x4(a, ad + r * 64u + ((p ^ ((r >> 1) & 3u)) << 4));
#pragma unroll
          for (int n = 0; n < NB; ++n) {
            if (bf) mma_bf16_16816(acc[m][n], a, b[n][2 * j], b[n][2 * j + 1]);
            else mma_f16_16816(acc[m][n], a, b[n][2 * j], b[n][2 * j + 1]);
          }
        }
      }
    }
    cp_async_wait_all();
    __syncthreads();                       // the rings are done with: the sums go over them
    float *mp = part + w * (ROWS * COLS);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        float *dp = mp + (16 * m + (l >> 2)) * COLS + 8 * n + 2 * (l & 3u);
        *reinterpret_cast<float2 *>(dp) = make_float2(acc[m][n][0], acc[m][n][1]);
        *reinterpret_cast<float2 *>(dp + 8 * COLS) = make_float2(acc[m][n][2], acc[m][n][3]);
      }
    __syncthreads();
    const uint32_t live = min(groups, kSkWarps);
#pragma unroll 1
    for (uint32_t e = L.tid; e < ROWS * COLS; e += 512u) {
      const uint32_t r = e / COLS, c = c0 + e % COLS;
      if (r >= M || c >= N) continue;
      float v = part[e];
#pragma unroll 4
      for (uint32_t s = 1; s < live; ++s) v += part[s * (ROWS * COLS) + e];
      if (out0) storef(out0, g.dt0, static_cast<int64_t>(r) * N + c, g.dt0 == kF32 ? v : quantize(v, g.qdt));
      v = sg_epilogue(g, res, v, r, c, csum);
      if (out1) storef(out1, g.dt1, mv ? at + view_index(mv->view, r * N + c) : static_cast<int64_t>(r) * N + c, v);
    }
  }
}

template <bool NORM>
__device__ __forceinline__ void skinny_shape(const Lane &L, const DSgemm &g, uint32_t slot, uint32_t n_slots, float &csum) {
  switch (g.shape) {           // 16-row blocks (1, 2) x 8-column blocks (1, 2, 4)
    case 0: skinny_run<1, 1, NORM>(L, g, slot, n_slots, csum); break;
    case 1: skinny_run<1, 2, NORM>(L, g, slot, n_slots, csum); break;
    case 2: skinny_run<1, 4, NORM>(L, g, slot, n_slots, csum); break;
    case 3: skinny_run<2, 1, NORM>(L, g, slot, n_slots, csum); break;
    case 4: skinny_run<2, 2, NORM>(L, g, slot, n_slots, csum); break;
    default: skinny_run<2, 4, NORM>(L, g, slot, n_slots, csum); break;
  }
}
static __device__ __noinline__ void skinny_tiles(const Lane &L, const DTask &t, uint32_t slot, uint32_t n_slots) {
  const DSgemm &g = *reinterpret_cast<const DSgemm *>(planned_desc(L, t));
  float csum = 0.0f;
  if (g.gamma) skinny_shape<true>(L, g, slot, n_slots, csum);
  else skinny_shape<false>(L, g, slot, n_slots, csum);
  if (g.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(*L.P, g.total)), t.p[3], g.n_owner_lanes);
}

}  // namespace b2
#endif
