// Matmuls of re-planned programs on the tensor cores (kTopGemm): bf16 / f16 operands, f32 accumulation in tensor memory,
// one or several products per task, and what followed the product elementwise as its store epilogue.
//
// Bound: the tensor pipe, under the power cap. What stood in its way in the tile op of the wire programs (ops_mma_tc.cuh,
// 830 TFLOP/s at 4096 cubed) is the issue of copies: one thread starts a TMA box every ~270 cycles whatever its size, and
// a 128 x 256 tile took up to six per 512 tensor cycles. Here a stage is two boxes (32 KB each at most) and feeds 1024.
// A 256 x 256 tile is two 128-row halves that share the B block and fill all of tensor memory.
//
// Roles: warp 0 feeds the stages (3 x 64 KB: A 256 x 64 k, B 256 x 64 k, each as 64 x 64 TMA boxes of 8 KB in the
// 128-byte swizzle, either operand k-contiguous or row / column-contiguous); warp 1 issues tcgen05.mma, the whole warp in
// step (its waits too: tc_wait_uniform) and one elected lane issuing, so that descriptors stay in uniform registers; warps
// 4-15 drain and store.
// Accumulator slots: a half tile takes slot (running number) % 2. A tile of one half thus runs under the previous one's
// epilogue; a tile of two halves starts its first half's k blocks as soon as that slot is drained, as far ahead as
// the stages reach, while the second slot drains.
// Tiles of a task are numbered product after product; lane slot i of n takes tiles i, i + n, ... (neighbouring lanes
// work on neighbouring tiles, which share operand blocks in L2), columns of a tile grid in groups of kGemmGroup rows.
#ifndef B2VM_OPS_GEMM_CUH_
#define B2VM_OPS_GEMM_CUH_

#include "dev_common.cuh"
#include "ops_ew.cuh"
#include "ops_fuse.cuh"
#include "plan_format.h"
#include "tc_common.cuh"

namespace b2 {

constexpr int kGemmStages = 3;
constexpr uint32_t kGemmStageBytes = 65536, kGemmBOff = 32768, kGemmBox = 8192;
constexpr uint32_t kGemmEpiWarps = 12, kGemmEpiFirst = 4;
constexpr uint32_t kGemmSlab = 32u * 64u;                  // staging of one epilogue warp: 32 rows x 64 bytes, 64-byte swizzle
constexpr uint32_t kGemmGroup = 8;

struct GemmShared {
  uint64_t full[kGemmStages], empty[kGemmStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base, failed;
};
static_assert(sizeof(GemmShared) <= 512, "fits the scratch slot");

// A tile: its product and place. Every role walks the lane's tiles with this.
struct GemmTile { uint32_t prob, r0, c0, halves, n_inst; };
__device__ __forceinline__ bool gemm_tile(const DGemm &g, uint32_t tile, GemmTile &o) {
  if (tile >= g.tiles) return false;
  uint32_t p = 0;
  while (p + 1u < g.n_prob && tile >= g.prob[p + 1u].first) ++p;
  const DGemmProb &q = g.prob[p];
  const uint32_t t = tile - q.first, per = kGemmGroup * q.tn, grp = t / per, in = t % per;
  const uint32_t rows = min(kGemmGroup, q.tm - grp * kGemmGroup);
  const uint32_t ti = grp * kGemmGroup + in % rows, tj = in / rows;
  o.prob = p;
  o.r0 = ti * (128u * q.halves);
  o.c0 = tj * q.bn;
  o.halves = q.halves == 2u && o.r0 + 128u < q.M ? 2u : 1u;
  o.n_inst = min(q.bn, (q.N - o.c0 + 15u) & ~15u);
  return true;
}

// The store epilogue on 32 consecutive columns of one row (plan_format.h: GemmEpi), in place.
struct GemmEpi {
  uint32_t flags, qdt, rdt;
  float s0, s1, gg;
  const uint8_t *res;
};
__device__ __forceinline__ void gemm_quant(float (&v)[32], uint32_t dt) {
  if (dt == kBF16) {
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const uint32_t w = cvt_bf16x2(v[j + 1], v[j]);
      v[j] = __uint_as_float(w << 16);
      v[j + 1] = __uint_as_float(w & 0xffff0000u);
    }
  } else if (dt == kF16) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = f16_bits_to_f32(f32_to_f16_bits(v[j]));
  }
}
// Eight residual elements from memory (ragged edge, or f32); else they come out of a prefetched 16-byte word.
__device__ __forceinline__ void gemm_res8(const uint8_t *row, uint32_t dt, uint32_t c, uint32_t left, float (&y)[8]) {
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) y[k] = k < left ? loadf(row, dt, static_cast<int64_t>(c) + k) : 0.0f;
}
__device__ __forceinline__ void gemm_epilogue(const GemmEpi &E, float (&v)[32], const uint8_t *res_row, const uint4 (&pre)[4], bool have_pre, uint32_t c,
                                              uint32_t left, bool row_ok, float &csum) {
  if (E.flags & kGeGelu) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
  }
  if (E.flags & kGeScale0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __fmul_rn(v[j], E.s0);
  }
  if (E.flags & kGeMaxS) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = np_max(v[j], E.s1);
  }
  if (E.flags & kGeRes) {
    const uint32_t op = E.flags & kGeResMask;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float y[8];
      if (have_pre) unpack8(pre[b], E.rdt, y);
      else if (row_ok) gemm_res8(res_row, E.rdt, c + 8u * b, left > 8u * b ? left - 8u * b : 0u, y);
      else {
#pragma unroll
        for (int k = 0; k < 8; ++k) y[k] = 0.0f;
      }
      float *w = &v[8 * b];
      if (op == kGeResAdd) {
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __fadd_rn(w[k], y[k]);
      } else if (op == kGeResSub) {
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __fsub_rn(w[k], y[k]);
      } else if (op == kGeResRSub) {
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __fsub_rn(y[k], w[k]);
      } else if (op == kGeResMul) {
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __fmul_rn(w[k], y[k]);
      } else {      // kGeResGeluGrad: times the derivative of tanh-GELU at the residual
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = __fmul_rn(w[k], gelu_grad(y[k], E.gg));
      }
    }
  }
  if (E.flags & kGeCarrySq) {
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 32; ++j) if (row_ok && static_cast<uint32_t>(j) < left) a[j & 3] = __fadd_rn(a[j & 3], __fmul_rn(v[j], v[j]));
    csum += (a[0] + a[1]) + (a[2] + a[3]);
  }
  if (E.flags & kGeScale1) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __fmul_rn(v[j], E.s1);
  }
}

// A warp's 32 x 32 block to its place. Each thread holds 32 columns of one row; stored like that, a warp instruction would
// touch 32 rows with 16 bytes each. Through the warp's slab (4 16-byte shared writes and reads per thread and pass, free of
// bank conflicts by the swizzle) it leaves as whole 64-byte row pieces, 8 rows per instruction. (The store unit out of
// the slab instead: the wait for the slab's previous box costs as much as it saves.)
__device__ __forceinline__ void gemm_store(uint8_t *dst, uint32_t dt, uint32_t N, uint32_t r_first, uint32_t M, uint32_t c, uint32_t left, bool vec,
                                           uint32_t stg, uint32_t lane, const float (&v)[32]) {
  if (left == 0u) return;
  const uint32_t esz = dt == kF32 ? 4u : 2u;
  if (vec && left == 32u) {
    const uint32_t row = stg + lane * 64u, sw = (lane >> 1) & 3u, r8 = lane >> 2, ch = lane & 3u;
#pragma unroll
    for (uint32_t h = 0; h < 2u; ++h) {                    // 16 columns of f32 fill the 64 bytes
      if (h == 1u && esz == 2u) break;
      __syncwarp();
#pragma unroll
      for (uint32_t k = 0; k < 4u; ++k) {
        uint32_t w[4];
        if (esz == 4u) {
#pragma unroll
          for (uint32_t e = 0; e < 4u; ++e) w[e] = __float_as_uint(h ? v[16 + 4 * k + e] : v[4 * k + e]);
        } else {
#pragma unroll
          for (uint32_t e = 0; e < 4u; ++e) {
            const float lo = v[8 * k + 2 * e], hi = v[8 * k + 2 * e + 1];
            w[e] = dt == kBF16 ? cvt_bf16x2(hi, lo) : (f32_to_f16_bits(lo) | (f32_to_f16_bits(hi) << 16));
          }
        }
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(row + ((k ^ sw) << 4)), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
      }
      __syncwarp();
      uint8_t *out = dst + (static_cast<size_t>(r_first + r8) * N + c) * esz + h * 64u + ch * 16u;
      const size_t step = static_cast<size_t>(8u) * N * esz;
#pragma unroll
      for (uint32_t p = 0; p < 4u; ++p) {
        const uint32_t rr = 8u * p + r8;
        uint4 w;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(stg + rr * 64u + ((ch ^ ((rr >> 1) & 3u)) << 4)) : "memory");
        if (r_first + rr < M) stg_v4(out + p * step, w);
      }
    }
    return;
  }
  const uint32_t rr = r_first + lane;
  if (rr >= M) return;
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (static_cast<uint32_t>(j) < left) storef(dst, dt, static_cast<int64_t>(rr) * N + c + j, v[j]);
}

static __device__ __noinline__ void gemm_tiles(const Lane &L, const DTask &t, uint32_t slot, uint32_t n_slots) {
  const KParams &P = *L.P;
  const DGemm &G = *reinterpret_cast<const DGemm *>(planned_desc(L, t));
  B2_DYN_SMEM(sm);
  GemmShared *S = reinterpret_cast<GemmShared *>(sm + kSmemRed);
  volatile uint32_t *failed = &S->failed;
  const uint32_t stage0 = (smem_addr(sm + kSmemSys) + 1023u) & ~1023u;
  const uint32_t w = __shfl_sync(0xffffffffu, L.tid / kWarp, 0), lane = L.tid % kWarp;   // the warp index, provably uniform
  const unsigned long long budget = P.wait_budget_ns;
  if (L.tid == 0) {
    for (int s = 0; s < kGemmStages; ++s) { mbar_init(&S->full[s], 1u); mbar_init(&S->empty[s], 1u); }
    for (int b = 0; b < 2; ++b) { mbar_init(&S->acc_full[b], 1u); mbar_init(&S->acc_empty[b], kGemmEpiWarps); }
    S->failed = 0u;
    fence_mbar_init();
  }
  __syncwarp();
  if (w == 2u) tmem_alloc(&S->tmem_base, 512u);
  fence_proxy_async_smem();   // what the entry before wrote here by ordinary stores, before asynchronous copies overwrite it
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = S->tmem_base;
  float csum = 0.0f;

  if (w == 0u) {
    // ---------------- producer ----------------
    if (lane == 0u) {
      fence_proxy_async_global();        // operands written by the previous phase's ordinary stores
      uint32_t it = 0;
      bool ok = true;
      GemmTile q;
      for (uint32_t tile = slot; ok && gemm_tile(G, tile, q); tile += n_slots) {
        const DGemmProb &pr = G.prob[q.prob];
        const DTmap *ta = P.tmaps + pr.tmap, *tb = ta + 1;
        const uint32_t nkb = (pr.K + 63u) / 64u, a_rows = 128u * pr.halves;
        const uint32_t bytes = (a_rows + pr.bn) * 128u;
        const int32_t r0 = static_cast<int32_t>(q.r0), c0 = static_cast<int32_t>(q.c0);
        // An operand's part of a stage is one box; one whose rows are the unit-stride axis comes as 64-row blocks (a box over
        // the blocks), or block by block where they do not divide the axis.
        auto fetch = [&](uint32_t dst, const DTmap *tm, uint32_t mode, uint32_t rows, int32_t r, int32_t k0, uint64_t *bar) {
          if (mode == kGmK) tma_load_3d(dst, tm, k0, r, 0, bar);
          else if (mode == kGmMnBlocks) tma_load_3d(dst, tm, 0, k0, r / 64, bar);
          else
            for (uint32_t i = 0; i < rows / 64u; ++i) tma_load_3d(dst + i * kGemmBox, tm, r + static_cast<int32_t>(64u * i), k0, 0, bar);
        };
        for (uint32_t kb = 0; kb < nkb; ++kb, ++it) {
          const uint32_t s = it % kGemmStages;
          if (!tc_wait(&S->empty[s], ((it / kGemmStages) & 1u) ^ 1u, failed, budget)) { ok = false; break; }
          mbar_arrive_tx(&S->full[s], bytes);
          const uint32_t sa = stage0 + s * kGemmStageBytes;
          const int32_t k0 = static_cast<int32_t>(kb * 64u);
          fetch(sa, ta, pr.amn, a_rows, r0, k0, &S->full[s]);
          fetch(sa + kGemmBOff, tb, pr.bmn, pr.bn, c0, k0, &S->full[s]);
        }
      }
      if (ok) tc_drain(S->empty, kGemmStages, it, failed, budget);
    }
  } else if (w == 1u) {
    // ---------------- issuer: the whole warp in step, one elected lane issuing ----------------
    uint32_t it = 0, n = 0;                         // stages consumed; accumulator slots taken
    bool ok = true;
    GemmTile q;
    __syncwarp();
    const bool leader = elect_one_sync();
    for (uint32_t tile = slot; ok && gemm_tile(G, tile, q); tile += n_slots) {
      const DGemmProb &pr = G.prob[q.prob];
      const uint32_t nkb = (pr.K + 63u) / 64u, fmt = pr.adt == kBF16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((pr.amn ? 1u : 0u) << 15) | ((pr.bmn ? 1u : 0u) << 16) |
                             ((q.n_inst >> 3) << 17) | ((128u >> 4) << 24);
      const uint64_t a_base = pr.amn ? tc_desc(stage0, 8192u, 1024u) : tc_desc(stage0, 16u, 1024u);
      const uint64_t b_base = pr.bmn ? tc_desc(stage0 + kGemmBOff, 8192u, 1024u) : tc_desc(stage0 + kGemmBOff, 16u, 1024u);
      const uint64_t adv_a = pr.amn ? (2048u >> 4) : (32u >> 4), adv_b = pr.bmn ? (2048u >> 4) : (32u >> 4);
      const uint32_t slot0 = n & 1u, slot1 = (n + 1u) & 1u;
      auto mma = [&](uint32_t s, uint32_t h, uint32_t kb) {
        const uint64_t da = a_base + static_cast<uint64_t>((s * kGemmStageBytes + h * 16384u) >> 4), db = b_base + static_cast<uint64_t>((s * kGemmStageBytes) >> 4);
        const uint32_t d = tmem + (h ? slot1 : slot0) * 256u;
        if (leader) {
#pragma unroll
          for (uint32_t j = 0; j < 4u; ++j) tc_mma_f16(d, da + j * adv_a, db + j * adv_b, idesc, (kb > 0u || j > 0u) ? 1u : 0u);
        }
      };
      auto drained = [&](uint32_t num) {            // accumulator slot of running number `num` is free
        const bool f = tc_wait_uniform(&S->acc_empty[num & 1u], ((num >> 1) & 1u) ^ 1u, failed, budget);
        tc_fence_after_sync();
        return f;
      };
      ok = drained(n);
      uint32_t kb = 0;
      if (ok && q.halves == 2u) {
        // the first half runs ahead over the stages that are there while the second slot drains
        const uint32_t ahead = min(nkb, static_cast<uint32_t>(kGemmStages));
        for (uint32_t i = 0; ok && i < ahead; ++i) {
          const uint32_t s = (it + i) % kGemmStages;
          ok = tc_wait_uniform(&S->full[s], ((it + i) / kGemmStages) & 1u, failed, budget);
          tc_fence_after_sync();
          if (ok) mma(s, 0u, i);
        }
        if (ok && ahead == nkb && leader) tc_commit(&S->acc_full[slot0]);
        ok = ok && drained(n + 1u);
        for (uint32_t i = 0; ok && i < ahead; ++i) {
          const uint32_t s = (it + i) % kGemmStages;
          mma(s, 1u, i);
          if (leader) tc_commit(&S->empty[s]);
        }
        kb = ahead;
        it += ahead;
      }
      for (; ok && kb < nkb; ++kb, ++it) {
        const uint32_t s = it % kGemmStages;
        ok = tc_wait_uniform(&S->full[s], (it / kGemmStages) & 1u, failed, budget);
        tc_fence_after_sync();
        if (!ok) break;
        mma(s, 0u, kb);
        if (kb + 1u == nkb && leader) tc_commit(&S->acc_full[slot0]);
        if (q.halves == 2u) mma(s, 1u, kb);
        if (leader) tc_commit(&S->empty[s]);
      }
      if (ok && q.halves == 2u && leader) tc_commit(&S->acc_full[slot1]);
      n += q.halves;
    }
  } else if (w >= kGemmEpiFirst) {
    // ---------------- epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. + 31; three warps share a quarter's column chunks ----------------
    const uint32_t ew = w - kGemmEpiFirst, quarter = w & 3u, third = ew >> 2;
    const uint32_t stg = stage0 + kGemmStages * kGemmStageBytes + ew * kGemmSlab;
    uint32_t n = 0;
    bool ok = true;
    GemmTile q;
    for (uint32_t tile = slot; ok && gemm_tile(G, tile, q); tile += n_slots) {
      const DGemmProb &pr = G.prob[q.prob];
      GemmEpi E;
      E.flags = pr.epi; E.qdt = pr.qdt; E.rdt = pr.rdt; E.s0 = pr.s0; E.s1 = pr.s1; E.gg = pr.gg;
      E.res = (pr.epi & kGeRes) ? resolve(P, pr.res) : nullptr;
      uint8_t *out0 = pr.out0 ? resolve(P, pr.out0) : nullptr, *out1 = pr.out1 ? resolve(P, pr.out1) : nullptr;
      const uint32_t M = pr.M, N = pr.N;
      const bool vec = (N & 7u) == 0u;                                    // 16-byte pieces of a row start on 16-byte boundaries
      const bool pre_ok = E.res && E.rdt != kF32 && vec;       // residual by 16-byte words, a chunk ahead
      for (uint32_t h = 0; ok && h < q.halves; ++h, ++n) {
        const uint32_t sl = n & 1u;
        const uint32_t rf = q.r0 + 128u * h + 32u * quarter, r = rf + lane;
        const bool row_ok = r < M;
        const uint8_t *res_row = E.res ? E.res + static_cast<size_t>(min(r, M - 1u)) * N * (E.rdt == kF32 ? 4u : 2u) : nullptr;
        uint4 nxt[4];
        auto prefetch = [&](uint32_t col) {
          const uint32_t c = q.c0 + col;
#pragma unroll
          for (uint32_t k = 0; k < 4u; ++k)
            nxt[k] = row_ok && c + 8u * k < N ? ldg_v4(res_row + static_cast<size_t>(c + 8u * k) * 2u) : make_uint4(0u, 0u, 0u, 0u);
        };
        if (pre_ok && 32u * third < q.n_inst) prefetch(32u * third);
        if (!tc_wait_warp(&S->acc_full[sl], (n >> 1) & 1u, failed, budget, 32u)) { ok = false; break; }
        tc_fence_after_sync();
#pragma unroll 1
        for (uint32_t col = 32u * third; col < q.n_inst; col += 96u) {
          uint32_t raw[32];
          __syncwarp();
          tc_ld32(tmem + ((32u * quarter) << 16) + sl * 256u + col, raw);
          uint4 cur[4];
          if (pre_ok) {
#pragma unroll
            for (int k = 0; k < 4; ++k) cur[k] = nxt[k];
            if (col + 96u < q.n_inst) prefetch(col + 96u);
          }
          tc_wait_ld();
          const uint32_t c = q.c0 + col, left = c < N ? min(32u, N - c) : 0u;
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
          if (E.flags & kGeQuant0) gemm_quant(v, E.qdt);
          if (out0) gemm_store(out0, pr.dt0, N, rf, M, c, left, vec, stg, lane, v);
          gemm_epilogue(E, v, res_row, cur, pre_ok, c, left, row_ok, csum);
          if (out1) gemm_store(out1, pr.dt1, N, rf, M, c, left, vec, stg, lane, v);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0u) mbar_arrive(&S->acc_empty[sl]);          // the warp is done with the slot
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  const bool gave_up = S->failed != 0u;
  if (gave_up) {
    // copies and products of other roles may still be in flight; nothing they wait for is outstanding, so they end by
    // themselves within microseconds, before tensor memory goes back
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) nanosleep_ns(1000);
  }
  if (w == 2u) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512u);
  }
  if (L.tid == 0) {
    if (gave_up) set_status(P, kStTensorTimeout, L.lane, slot, kTopGemm);
    else {
      for (int s = 0; s < kGemmStages; ++s) { mbar_inval(&S->full[s]); mbar_inval(&S->empty[s]); }
      for (int b = 0; b < 2; ++b) { mbar_inval(&S->acc_full[b]); mbar_inval(&S->acc_empty[b]); }
    }
  }
  __syncthreads();
  if (G.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(P, G.total)), t.p[3], G.n_owner_lanes);
}

}  // namespace b2
#endif
