// Matmuls of re-planned programs on the tensor cores (kTopGemm): bf16 / f16 operands, f32 accumulation in tensor memory,
// one or several products per task, and what followed the product elementwise as its store epilogue.
//
// Bound: the tensor pipe, under the power cap. What stood in its way in the tile op of the wire programs (ops_mma_tc.cuh,
// 830 TFLOP/s at 4096 cubed) is the issue of copies: one thread starts a TMA box every ~270 cycles whatever its size, and
// a 128 x 256 tile took up to six per 512 tensor cycles. Here a stage is two boxes (32 KB each at most) and feeds 1024.
// A 256 x 256 tile is two 128-row halves that share the B block and fill all of tensor memory.
//
// Roles: two threads of warp 0 feed the stages, one for each operand (64 k of A's rows and of B's columns, as 64 x 64 TMA boxes of 8 KB
// in the 128-byte swizzle, either operand k-contiguous or row / column-contiguous; as many stages of the task's largest tile as the
// ring's 192 KB hold, 3 of 256 x 256, 4 of 128 x 256, 8 of 128 x 64); warp 1 issues tcgen05.mma, the whole warp in step (its waits
// too: tc_wait_uniform) and one elected lane issuing, so that descriptors stay in uniform registers; warps 4-15 drain and store.
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

constexpr uint32_t kGemmBox = 8192;
constexpr uint32_t kGemmEpiWarps = 12, kGemmEpiFirst = 4;
constexpr uint32_t kGemmSlab = 32u * 64u;                  // staging of one epilogue warp: 32 rows x 64 bytes, 64-byte swizzle
constexpr uint32_t kGemmGroup = 8;

struct GemmShared {
  uint64_t full[kGemmStagesMax], empty[kGemmStagesMax];
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

// How the general epilogue gets its residual: not at all, by prefetched 16-byte words, or element by element (f32, ragged rows). Each is
// a function of its own: the words' registers would be missing in the others (a 16-bit product that leaves as f32, 4096 x 4096 by K =
// 1024: 60 us with all in one, 50 so; 52 when the epilogue was part of gemm_tiles).
enum GemmRes : uint32_t { kGrNone, kGrWords, kGrElems };
struct GemmEpi { uint32_t epi, qdt, rdt; float s0, s1, gg; };
__device__ __forceinline__ GemmRes gemm_res_of(const DGemmProb &pr) {
  return !(pr.epi & kGeRes) ? kGrNone : pr.rdt != kF32 && (pr.N & 7u) == 0u ? kGrWords : kGrElems;
}
// The store epilogue on 32 consecutive columns of one row (plan_format.h: GemmEpi), in place.
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
  if (dt == kF32) {
    const float *p = reinterpret_cast<const float *>(row) + c;
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k) y[k] = k < left ? p[k] : 0.0f;
  } else {
    const uint16_t *p = reinterpret_cast<const uint16_t *>(row) + c;
#pragma unroll
    for (uint32_t k = 0; k < 8u; ++k) {
      const uint32_t x = k < left ? p[k] : 0u;
      y[k] = dt == kBF16 ? bf16_bits_to_f32(x) : f16_bits_to_f32(x);
    }
  }
}
template <GemmRes RES, typename Epi>
__device__ __forceinline__ void gemm_epilogue(const Epi &E, float (&v)[32], const uint8_t *res_row, uint32_t stg, uint32_t lane, uint32_t c, uint32_t left,
                                              bool row_ok, float &csum) {
  if (E.epi & kGeGelu) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
  }
  if (E.epi & kGeScale0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __fmul_rn(v[j], E.s0);
  }
  if (E.epi & kGeMaxS) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = np_max(v[j], E.s1);
  }
  if constexpr (RES != kGrNone) {
    const uint32_t op = E.epi & kGeResMask;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float y[8];
      if (RES == kGrWords) unpack8(lds_v4(stg + lane * 64u + ((static_cast<uint32_t>(b) ^ ((lane >> 1) & 3u)) << 4)), E.rdt, y);
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
  if (E.epi & kGeCarrySq) {
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 32; ++j) if (row_ok && static_cast<uint32_t>(j) < left) a[j & 3] = __fadd_rn(a[j & 3], __fmul_rn(v[j], v[j]));
    csum += (a[0] + a[1]) + (a[2] + a[3]);
  }
  if (E.epi & kGeScale1) {
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
  if (vec) {                                               // (and then whole 16-byte pieces are all there is)
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
        if (r_first + rr < M && h * 16u + ch * (16u / esz) < left) stg_v4(out + p * step, w);
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

// ---- the epilogue warps: warp w reads tensor-memory lanes 32 (w % 4) .. + 31; three warps share a quarter's 32-column chunks ----
// Where a warp stands: its next tile, half tiles done, its share of the full sum.
struct GemmAt { uint32_t tile, n; float csum; bool ok; };
// What the warp works with.
struct GemmWarp {
  const KParams *P;
  uint32_t tmem, n_slots, stg, quarter, third, lane;
};
// The task's descriptor and barriers, at fixed places of the lane's shared memory.
__device__ __forceinline__ const DGemm &gemm_desc() { B2_DYN_SMEM(sm); return *reinterpret_cast<const DGemm *>(sm + kSmemDesc); }
__device__ __forceinline__ GemmShared *gemm_shared() { B2_DYN_SMEM(sm); return reinterpret_cast<GemmShared *>(sm + kSmemRed); }
// The accumulator slot of half tile `n` is full; the warp is done with it.
__device__ __forceinline__ bool gemm_slot_full(const GemmWarp &W, uint32_t n) {
  const bool f = tc_wait_warp(&gemm_shared()->acc_full[n & 1u], (n >> 1) & 1u, &gemm_shared()->failed, W.P->wait_budget_ns, 32u);
  tc_fence_after_sync();
  return f;
}
__device__ __forceinline__ void gemm_slot_done(const GemmWarp &W, uint32_t n) {
  tc_fence_before_sync();
  __syncwarp();
  if (W.lane == 0u) mbar_arrive(&gemm_shared()->acc_empty[n & 1u]);
}

// Any epilogue, its steps looked at chunk by chunk; the warp's tiles from `at` on as long as they want this.
template <GemmRes RES>
static __device__ __noinline__ GemmAt gemm_form_any(GemmWarp W, GemmAt at) {
  const DGemm &G = gemm_desc();
  const KParams &P = *W.P;
  const uint32_t lane = W.lane, r8 = lane >> 2, ch = lane & 3u, piece = W.stg + r8 * 64u + ((ch ^ ((r8 >> 1) & 3u)) << 4);
  GemmTile q;
  for (; at.ok && gemm_tile(G, at.tile, q) && G.prob[q.prob].form == kGfAny && gemm_res_of(G.prob[q.prob]) == RES; at.tile += W.n_slots) {
    const DGemmProb &pr = G.prob[q.prob];
    const GemmEpi own = {pr.epi, pr.qdt, pr.rdt, pr.s0, pr.s1, pr.gg};
    // With the words' registers there are none to keep these in: they are read where they are wanted (78 us for 72, 8192 x 1024 by K = 4096
    // times a 16-bit array; without the words 199 us for 205, 4096 x 4100 by K = 1024).
    const auto &E = [&]() -> const auto & { if constexpr (RES == kGrWords) return pr; else return own; }();
    const uint8_t *res = RES != kGrNone ? resolve(P, pr.res) : nullptr;
    uint8_t *out0 = pr.out0 ? resolve(P, pr.out0) : nullptr, *out1 = pr.out1 ? resolve(P, pr.out1) : nullptr;
    const uint32_t M = pr.M, N = pr.N;
    const bool vec = RES == kGrWords || (N & 7u) == 0u;                 // 16-byte pieces of a row start on 16-byte boundaries
    for (uint32_t h = 0; h < q.halves; ++h, ++at.n) {
      const uint32_t rf = q.r0 + 128u * h + 32u * W.quarter, r = rf + lane, acc = W.tmem + ((32u * W.quarter) << 16) + (at.n & 1u) * 256u;
      const bool row_ok = r < M;
      const uint8_t *res_row = RES == kGrElems ? res + static_cast<size_t>(min(r, M - 1u)) * N * (E.rdt == kF32 ? 4u : 2u) : nullptr;
      const uint32_t rows = M > rf + r8 ? (M - rf - r8 + 7u) / 8u : 0u;               // of this thread's four row pieces
      uint4 nxt[4];                                          // the residual's words, a chunk ahead: 64-byte pieces of four rows
      auto prefetch = [&](uint32_t col) {
        const uint8_t *src = res + (static_cast<size_t>(rf + r8) * N + q.c0 + col + 8u * ch) * 2u;
#pragma unroll
        for (uint32_t p = 0; p < 4u; ++p)
          nxt[p] = p < rows && q.c0 + col + 8u * ch < N ? ldg_v4(src + static_cast<size_t>(p) * N * 16u) : make_uint4(0u, 0u, 0u, 0u);
      };
      if (RES == kGrWords && 32u * W.third < q.n_inst) prefetch(32u * W.third);
      if (!gemm_slot_full(W, at.n)) { at.ok = false; return at; }
#pragma unroll 1
      for (uint32_t col = 32u * W.third; col < q.n_inst; col += 96u) {
        uint32_t raw[32];
        __syncwarp();
        tc_ld32(acc + col, raw);
        tc_wait_ld();
        const uint32_t c = q.c0 + col, left = c < N ? min(32u, N - c) : 0u;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
        if (E.epi & kGeQuant0) gemm_quant(v, E.qdt);
        if (out0) gemm_store(out0, pr.dt0, N, rf, M, c, left, vec, W.stg, lane, v);
        if (RES == kGrWords) {
          __syncwarp();
#pragma unroll
          for (uint32_t p = 0; p < 4u; ++p) sts_v4(piece + 512u * p, nxt[p]);
          if (col + 96u < q.n_inst) prefetch(col + 96u);
          __syncwarp();
        }
        gemm_epilogue<RES>(E, v, res_row, W.stg, lane, c, left, row_ok, at.csum);
        if (RES == kGrWords) __syncwarp();
        if (out1) gemm_store(out1, pr.dt1, N, rf, M, c, left, vec, W.stg, lane, v);
      }
      gemm_slot_done(W, at.n);
    }
  }
  return at;
}

// An epilogue whose steps are known when this is compiled: FL = its flags but for kGeQuant0, every value that is stored or
// read 16-bit of one type (BF: bf16), rows whole 16-byte words. Such a form is a function of its own, entered once for all of the
// warp's tiles in a row that want it, so that what a chunk needs stays in registers: the lane's shared memory leaves hardly any
// L1, every use of a spilled value is a trip to L2, and the general form has its steps as branches and predicates. A 256 x 256
// tile that only leaves as bf16 takes 7000 cycles here, 22000 with all steps in one function (2 tiles of K = 64: 31 us, now 15.5); what is left
// is mostly the SM's way to L2, 32 bytes a cycle. Rows of the residual come as the result goes: whole 64-byte row pieces through the
// warp's slab, a chunk ahead. Tried: all of a tile's chunks held in registers first and stored when the slots are given back
// (more code and registers, slower: 110 us against 107 for 16384 x 4096 by K = 1024); 32-byte stores from the rows as they come
// (an SM then sends 17 bytes a cycle).
template <bool BF>
__device__ __forceinline__ uint32_t gemm_pack(float lo, float hi) { return BF ? cvt_bf16x2(hi, lo) : cvt_f16x2(hi, lo); }
template <uint32_t FORM, uint32_t FL, bool BF>
static __device__ __noinline__ GemmAt gemm_form(GemmWarp W, GemmAt at) {
  constexpr uint32_t dt = BF ? static_cast<uint32_t>(kBF16) : static_cast<uint32_t>(kF16);
  constexpr bool kRes = (FL & kGeRes) != 0u;
  const DGemm &G = gemm_desc();
  const uint32_t lane = W.lane, sw = (lane >> 1) & 3u, row = W.stg + lane * 64u, r8 = lane >> 2, ch = lane & 3u;
  const uint32_t piece = W.stg + r8 * 64u + ((ch ^ ((r8 >> 1) & 3u)) << 4);          // + 512 p: row 8 p + r8
  GemmTile q;
  for (; gemm_tile(G, at.tile, q) && G.prob[q.prob].form == FORM; at.tile += W.n_slots) {
    const DGemmProb &pr = G.prob[q.prob];
    const uint32_t M = pr.M, N = pr.N;
    const bool quant = (pr.epi & kGeQuant0) != 0u;
    const float s0 = pr.s0, s1 = pr.s1, gg = pr.gg;
    const uint8_t *res = kRes ? resolve(*W.P, pr.res) : nullptr;
    uint8_t *out0 = FL == kGeGelu && pr.out0 ? resolve(*W.P, pr.out0) : nullptr, *out1 = resolve(*W.P, pr.out1);
    for (uint32_t h = 0; h < q.halves; ++h, ++at.n) {
      const uint32_t rf = q.r0 + 128u * h + 32u * W.quarter, acc = W.tmem + ((32u * W.quarter) << 16) + (at.n & 1u) * 256u;
      const uint32_t rows = M > rf + r8 ? (M - rf - r8 + 7u) / 8u : 0u;               // of this thread's four row pieces
      const size_t first = (static_cast<size_t>(rf + r8) * N + q.c0 + 8u * ch) * 2u, step = static_cast<size_t>(N) * 16u;
      uint4 nxt[4] = {};
      auto prefetch = [&](uint32_t col) {
        const uint8_t *src = res + first + col * 2u;
#pragma unroll
        for (uint32_t p = 0; p < 4u; ++p)
          nxt[p] = p < rows && q.c0 + col + 8u * ch < N ? ldg_v4(src + p * step) : make_uint4(0u, 0u, 0u, 0u);
      };
      auto leave = [&](uint8_t *out, uint32_t col) {             // the slab to memory
        __syncwarp();
        uint8_t *dst = out + first + col * 2u;
        const uint32_t live = q.c0 + col + 8u * ch < N ? rows : 0u;
#pragma unroll
        for (uint32_t p = 0; p < 4u; ++p) {
          const uint4 x = lds_v4(piece + 512u * p);
          if (p < live) stg_v4(dst + p * step, x);
        }
        __syncwarp();
      };
      if (kRes && 32u * W.third < q.n_inst) prefetch(32u * W.third);
      if (!gemm_slot_full(W, at.n)) { at.ok = false; return at; }
      if (32u * W.third >= q.n_inst) gemm_slot_done(W, at.n);
#pragma unroll 1
      for (uint32_t col = 32u * W.third; col < q.n_inst; col += 96u) {
        uint32_t raw[32];
        __syncwarp();
        tc_ld32(acc + col, raw);
        if (kRes) {
#pragma unroll
          for (uint32_t p = 0; p < 4u; ++p) sts_v4(piece + 512u * p, nxt[p]);
          if (col + 96u < q.n_inst) prefetch(col + 96u);
          __syncwarp();
        }
        tc_wait_ld();
        if (col + 96u >= q.n_inst) gemm_slot_done(W, at.n);      // its last columns are in registers
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
        if (FL != 0u && quant) {                                 // (alone, the store rounds)
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            w[j] = gemm_pack<BF>(v[2 * j], v[2 * j + 1]);
            if (BF) { v[2 * j] = __uint_as_float(w[j] << 16); v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u); }
            else { v[2 * j] = f16_bits_to_f32(w[j] & 0xffffu); v[2 * j + 1] = f16_bits_to_f32(w[j] >> 16); }
          }
          if constexpr (FL == kGeGelu) {
            if (out0) {
#pragma unroll
              for (uint32_t k = 0; k < 4u; ++k) sts_v4(row + ((k ^ sw) << 4), make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]));
              leave(out0, col);
            }
          }
        }
        float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
          float *x = &v[8 * k];
          if constexpr ((FL & kGeGelu) != 0u) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = gelu_tanh(x[e]);
          }
          if constexpr ((FL & kGeScale0) != 0u) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = __fmul_rn(x[e], s0);
          }
          if constexpr (kRes) {
            constexpr uint32_t op = FL & kGeResMask;
            float y[8];
            unpack8(lds_v4(row + ((k ^ sw) << 4)), dt, y);
#pragma unroll
            for (int e = 0; e < 8; ++e)
              x[e] = op == kGeResAdd ? __fadd_rn(x[e], y[e]) : op == kGeResSub ? __fsub_rn(x[e], y[e]) : op == kGeResRSub ? __fsub_rn(y[e], x[e])
                   : __fmul_rn(x[e], gelu_grad(y[e], gg));
          }
          if constexpr ((FL & kGeCarrySq) != 0u) {
            if (rf + lane < M && q.c0 + col + 8u * k < N) {
#pragma unroll
              for (int e = 0; e < 8; ++e) part[e & 3] = __fadd_rn(part[e & 3], __fmul_rn(x[e], x[e]));
            }
          }
          if constexpr ((FL & kGeScale1) != 0u) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = __fmul_rn(x[e], s1);
          }
          sts_v4(row + ((k ^ sw) << 4), make_uint4(gemm_pack<BF>(x[0], x[1]), gemm_pack<BF>(x[2], x[3]), gemm_pack<BF>(x[4], x[5]), gemm_pack<BF>(x[6], x[7])));
        }
        if constexpr ((FL & kGeCarrySq) != 0u) at.csum += (part[0] + part[1]) + (part[2] + part[3]);
        leave(out1, col);
      }
    }
  }
  return at;
}

// ---- the warps that feed the tensor cores, each a function of its own: what they need per stage stays in registers ----
struct GemmLane { const KParams *P; uint32_t stage0, tmem, slot, n_slots; };
// Two threads, one for each operand: fill the stages. (A box takes its thread ~270 cycles to start; with both operands' boxes from one
// thread a stage of a small tile took 640-780, more than its products.)
static __device__ __noinline__ void gemm_produce(GemmLane X, uint32_t side) {
  const DGemm &G = gemm_desc();
  GemmShared *S = gemm_shared();
  volatile uint32_t *failed = &S->failed;
  const unsigned long long budget = X.P->wait_budget_ns;
  const uint32_t n_stages = G.stages, stage_bytes = G.stage_bytes;
  fence_proxy_async_global();        // operands written by the previous phase's ordinary stores
  uint32_t it = 0, s = 0, turn = 1u;         // stages filled; the next one, and the parity that it is empty with
  bool ok = true;
  GemmTile q;
  for (uint32_t tile = X.slot; ok && gemm_tile(G, tile, q); tile += X.n_slots) {
    const DGemmProb &pr = G.prob[q.prob];
    const DTmap *tm = X.P->tmaps + pr.tmap + side;
    const uint32_t nkb = (pr.K + 63u) / 64u, mode = side ? pr.bmn : pr.amn, rows = side ? pr.bn : 128u * pr.halves;
    const uint32_t bytes = rows * 128u, at = X.stage0 + (side ? 16384u * pr.halves : 0u);
    // An operand's part of a stage is one box; one whose rows are the unit-stride axis comes as 64-row blocks (a box over
    // the blocks), or block by block where they do not divide the axis.
    const int32_t r = static_cast<int32_t>(side ? q.c0 : q.r0);
    const int32_t dx = mode == kGmK ? 64 : 0, dy = mode == kGmK ? 0 : 64, z = mode == kGmMnBlocks ? r / 64 : 0;
    int32_t x = mode == kGmMnSingle ? r : 0, y = mode == kGmK ? r : 0;
    for (uint32_t kb = 0; kb < nkb; ++kb, ++it) {
      if (!tc_wait(&S->empty[s], turn, failed, budget)) { ok = false; break; }
      mbar_arrive_tx(&S->full[s], bytes);
      const uint32_t dst = at + s * stage_bytes;
      tma_load_3d(dst, tm, x, y, z, &S->full[s]);
      if (mode == kGmMnSingle)
        for (uint32_t i = 1; i < rows / 64u; ++i) tma_load_3d(dst + i * kGemmBox, tm, x + static_cast<int32_t>(64u * i), y, 0, &S->full[s]);
      x += dx;
      y += dy;
      if (++s == n_stages) { s = 0u; turn ^= 1u; }
    }
  }
  if (ok) tc_drain(S->empty, n_stages, it, failed, budget);
}
// A whole warp in step, one elected lane issuing.
static __device__ __noinline__ void gemm_issue(GemmLane X) {
  const DGemm &G = gemm_desc();
  GemmShared *S = gemm_shared();
  volatile uint32_t *failed = &S->failed;
  const unsigned long long budget = X.P->wait_budget_ns;
  const uint32_t n_stages = G.stages, stage_bytes = G.stage_bytes, stage0 = X.stage0, tmem = X.tmem;
  uint32_t s = 0, turn = 0, n = 0;                // the next stage, and the parity that it is full with; accumulator slots taken
  bool ok = true;
  GemmTile q;
  __syncwarp();
  const bool leader = elect_one_sync();
  for (uint32_t tile = X.slot; ok && gemm_tile(G, tile, q); tile += X.n_slots) {
    const DGemmProb &pr = G.prob[q.prob];
    const uint32_t nkb = (pr.K + 63u) / 64u, fmt = pr.adt == kBF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((pr.amn ? 1u : 0u) << 15) | ((pr.bmn ? 1u : 0u) << 16) |
                           ((q.n_inst >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t a_base = pr.amn ? tc_desc(stage0, 8192u, 1024u) : tc_desc(stage0, 16u, 1024u);
    const uint32_t b0 = stage0 + 16384u * pr.halves;
    const uint64_t b_base = pr.bmn ? tc_desc(b0, 8192u, 1024u) : tc_desc(b0, 16u, 1024u);
    const uint64_t adv_a = pr.amn ? (2048u >> 4) : (32u >> 4), adv_b = pr.bmn ? (2048u >> 4) : (32u >> 4);
    const uint32_t slot0 = n & 1u, slot1 = (n + 1u) & 1u;
    auto mma = [&](uint32_t s, uint32_t h, uint32_t kb) {
      const uint64_t da = a_base + static_cast<uint64_t>((s * stage_bytes + h * 16384u) >> 4), db = b_base + static_cast<uint64_t>((s * stage_bytes) >> 4);
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
    auto landed = [&](uint32_t st, uint32_t parity) {
      const bool f = tc_wait_uniform(&S->full[st], parity, failed, budget);
      tc_fence_after_sync();
      return f;
    };
    uint32_t kb = 0;
    if (ok && q.halves == 2u) {
      // the first half runs ahead over the stages that are there while the second slot drains
      const uint32_t ahead = min(nkb, n_stages);
      uint32_t s1 = s, turn1 = turn;
      for (uint32_t i = 0; ok && i < ahead; ++i) {
        ok = landed(s1, turn1);
        if (ok) mma(s1, 0u, i);
        if (++s1 == n_stages) { s1 = 0u; turn1 ^= 1u; }
      }
      if (ok && ahead == nkb && leader) tc_commit(&S->acc_full[slot0]);
      ok = ok && drained(n + 1u);
      for (uint32_t i = 0; ok && i < ahead; ++i) {
        mma(s, 1u, i);
        if (leader) tc_commit(&S->empty[s]);
        if (++s == n_stages) { s = 0u; turn ^= 1u; }
      }
      kb = ahead;
    }
    for (; ok && kb < nkb; ++kb) {
      ok = landed(s, turn);
      if (!ok) break;
      mma(s, 0u, kb);
      if (kb + 1u == nkb && leader) tc_commit(&S->acc_full[slot0]);
      if (q.halves == 2u) mma(s, 1u, kb);
      if (leader) tc_commit(&S->empty[s]);
      if (++s == n_stages) { s = 0u; turn ^= 1u; }
    }
    if (ok && q.halves == 2u && leader) tc_commit(&S->acc_full[slot1]);
    n += q.halves;
  }
}

static __device__ __noinline__ void gemm_tiles(const Lane &L, const DTask &t, uint32_t slot, uint32_t n_slots) {
  const KParams &P = *L.P;
  planned_desc(L, t);
  B2_DYN_SMEM(sm);
  const DGemm &G = gemm_desc();
  GemmShared *S = gemm_shared();
  const uint32_t stage0 = (smem_addr(sm + kSmemSys) + 1023u) & ~1023u;
  const uint32_t w = __shfl_sync(0xffffffffu, L.tid / kWarp, 0), lane = L.tid % kWarp;   // the warp index, provably uniform
  const uint32_t n_stages = G.stages;
  if (w == 0u) {
    if (lane < n_stages) { mbar_init(&S->full[lane], 2u); mbar_init(&S->empty[lane], 1u); }
    else if (lane < n_stages + 2u) { mbar_init(&S->acc_full[lane - n_stages], 1u); mbar_init(&S->acc_empty[lane - n_stages], kGemmEpiWarps); }
    else if (lane == 31u) S->failed = 0u;
    fence_mbar_init();
  } else if (w == 1u && lane < 2u * G.n_prob) {
    prefetch_tmap(P.tmaps + G.prob[lane >> 1].tmap + (lane & 1u));       // the first copy would wait for it
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
    if (lane < 2u) gemm_produce(GemmLane{&P, stage0, tmem, slot, n_slots}, lane);
  } else if (w == 1u) {
    gemm_issue(GemmLane{&P, stage0, tmem, slot, n_slots});
  } else if (w >= kGemmEpiFirst) {
    const uint32_t ew = w - kGemmEpiFirst;
    const GemmWarp W = {&P, tmem, n_slots, stage0 + kGemmRing + ew * kGemmSlab, w & 3u, ew >> 2, lane};
    GemmAt at = {slot, 0u, 0.0f, true};
    GemmTile q;
    while (at.ok && gemm_tile(G, at.tile, q)) {
      switch (G.prob[q.prob].form) {
#define B2_GEMM_FORM(f, flags)                                          \
        case f: at = gemm_form<f, flags, true>(W, at); break;           \
        case f + kGfF16: at = gemm_form<f + kGfF16, flags, false>(W, at); break;
        B2_GEMM_FORM(kGfPlain, 0u)
        B2_GEMM_FORM(kGfGelu, kGeGelu)
        B2_GEMM_FORM(kGfAdd, kGeRes | kGeResAdd)
        B2_GEMM_FORM(kGfGrad, kGeRes | kGeResGeluGrad)
        B2_GEMM_FORM(kGfStep, kGeScale0 | kGeRes | kGeResRSub)
        B2_GEMM_FORM(kGfLoss, kGeRes | kGeResSub | kGeCarrySq | kGeScale1)
#undef B2_GEMM_FORM
        default:
          switch (gemm_res_of(G.prob[q.prob])) {
            case kGrNone: at = gemm_form_any<kGrNone>(W, at); break;
            case kGrWords: at = gemm_form_any<kGrWords>(W, at); break;
            default: at = gemm_form_any<kGrElems>(W, at); break;
          }
          break;
      }
    }
    csum = at.csum;
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
  if (gave_up) {
    if (L.tid == 0) set_status(P, kStTensorTimeout, L.lane, slot, kTopGemm);
  } else if (w == 0u) {
    if (lane < n_stages) { mbar_inval(&S->full[lane]); mbar_inval(&S->empty[lane]); }
    else if (lane < n_stages + 2u) { mbar_inval(&S->acc_full[lane - n_stages]); mbar_inval(&S->acc_empty[lane - n_stages]); }
  }
  __syncthreads();
  if (G.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(P, G.total)), t.p[3], G.n_owner_lanes);
}

}  // namespace b2
#endif
