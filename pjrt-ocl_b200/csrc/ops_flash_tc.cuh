// TILE_FLASH_ATTN on the tensor cores: S = Q K^T and O = P V as tcgen05.mma with the
// accumulators in tensor memory, online softmax in between.
//
// Same contract as the CUDA-core path (ops_flash.cuh; pjrt_plugin/kernels/ops/
// attention.cl:49-159; python/pjrt_ocl/ops/attention.py:52-66): tile = one query row
// (head g, position m) of out[H,T,hd]; Q [H,T,hd], K given as the QK^T matmul's B
// operand [H,hd,C], V [H,C,hd], each possibly through a view; with `causal` key c is
// masked when c > m + C - T. Taken for bf16 / f16 operands with head_dim 64 whose
// (viewed) layouts three rank-4 TMA tensor maps can describe (DFlash::tc_mode; the
// loader decides), so a [batch, seq, heads, hd] projection is attended in place.
//
// Bound: latency. Of the units the exponentials' is the busiest: 16 a cycle and SM, 512 cycles for 128 rows x 64 keys, where the two
// products take ~330; it is 47 % busy (8 x 2048 causal, 16 heads: 141 us, 66 of them exponentials). A block takes a slot alone 1870
// cycles, three slots together 2750 for 1536 of exponentials. To fill them a lane works on three query tiles of 128 rows at a time ("slots"), independent of
// each other: each has its own softmax warps (one of each on every scheduler), its own feeding warp, its own Q, K and V in shared
// memory and its own columns of tensor memory, draws its own tiles, and waits for nobody else. (Two slots that shared one
// stream of 128-key blocks, one issuing warp looking after both and P in shared memory: 6300 cycles per block and slot, of which
// 3900 in two passes over the scores and 1050 waiting for P's buffer: 257 us of a block of 8 x 2048 with 16 heads.)
// Tiles are handed out heaviest first from a counter in the program's scratch when the loader allowed it (causal tiles differ
// 16 x in cost), else a lane's slots take turns over the tiles that start inside its row range.
// Per slot and block of 64 keys:
//   its feeding warp   TMA for Q once per tile, K and V by 64-key blocks through rings of three, each stage refilled as soon as
//            the product that read it is known to be done; S(j) = Q K(j)^T (128 x 64 x 64) as soon as the scores before are in
//            registers, so that they are there when the softmax comes back; O (+)= P(j-1) V(j-1) when P is written.
//   its four softmax warps, one thread per query row: the row's 64 scores into registers, their maximum, 2^(s - max) (log2
//            domain, one ex2 each), P as 16-bit values back into tensor memory, where the second product reads it.
//            O stays in tensor memory for the whole tile; it is rescaled in place only when a row's maximum grew by more
//            than 2^8 since the maximum in use was set - P then stays below 256 and the result is mathematically unchanged.
//            Finally out = O / (row sum).
// Every wait is bounded; a wait that runs out ends the task with a status.
#ifndef B2VM_OPS_FLASH_TC_CUH_
#define B2VM_OPS_FLASH_TC_CUH_

#include "ops_flash.cuh"
#include "ops_mma_tc.cuh"

namespace b2 {

#if B2_HAS_TC

constexpr uint32_t kFaSlots = 3, kFaStages = 3;
constexpr uint32_t kFaQ = 128 * 128, kFaKv = 64 * 128;          // bytes of a Q tile (128 x 64 x 2), a K or V block (64 x 64 x 2)
constexpr uint32_t kFaSlotCols = 160, kFaCols = 512;            // of a slot: S 0, O 64, P 128 (two values per column)
constexpr float kFaRescale = 8.0f;             // log2 of the growth of a row maximum that forces a rescale
constexpr uint32_t kFaNone = 0xffffffffu;

struct FaShared {
  uint64_t t_full[kFaSlots];                   // feed -> softmax: the slot's next tile is known
  uint64_t q_full[kFaSlots];
  uint64_t k_full[kFaSlots][kFaStages], v_full[kFaSlots][kFaStages];
  uint64_t s_full[kFaSlots];                   // product -> softmax: the slot's scores are in tensor memory
  uint64_t s_free[kFaSlots];                   // softmax -> feed: the scores have been read (4 warp arrivals)
  uint64_t p_full[kFaSlots];                   // softmax -> feed: P is in tensor memory, O is rescaled (4 warp arrivals)
  uint64_t pv_done[kFaSlots];                  // product -> softmax: O holds the block, P has been read
  uint32_t tile[kFaSlots][2];                  // by turns
  uint32_t tmem_base, failed;
};
// What every role needs to know of the task.
struct FaTask {
  const DTmap *tm_q;
  uint32_t *work;                              // dynamic: {next tile, lanes done}; else null
  uint8_t *out;
  unsigned long long budget;
  int32_t H, T, C, per_head;                   // tiles of 128 rows per head
  uint32_t first, stop;                        // static: the lane's tiles. dynamic: the lane, tiles that slots take first (or 0)
  uint32_t h0_size, causal, k_mn, adt, dt, base;
  float sl2;
};
// Both lie in the reduction scratch, which nothing else uses while the op runs: past it is the interpreter's (the task itself).
constexpr uint32_t kFaTaskAt = kSmemRed + (sizeof(FaShared) + 15u) / 16u * 16u;
static_assert(kFaTaskAt + sizeof(FaTask) <= static_cast<uint32_t>(kSmemPtrs), "fit the reduction scratch");
__device__ __forceinline__ FaShared *fa_shared() { B2_DYN_SMEM(sm); return reinterpret_cast<FaShared *>(sm + kSmemRed); }
__device__ __forceinline__ FaTask *fa_task() { B2_DYN_SMEM(sm); return reinterpret_cast<FaTask *>(sm + kFaTaskAt); }

// A tile: head, first row, blocks of keys that its rows may see.
struct FaTile { int32_t g, m0, blocks; };
__device__ __forceinline__ FaTile fa_tile(const FaTask &F, uint32_t u) {
  FaTile t;
  t.g = static_cast<int32_t>(u) / F.per_head;
  t.m0 = (static_cast<int32_t>(u) - t.g * F.per_head) * 128;
  const int32_t c_max = F.causal ? min(F.C, t.m0 + min(128, F.T - t.m0) + (F.C - F.T)) : F.C;
  t.blocks = c_max <= 0 ? 0 : (c_max + 63) / 64;
  return t;
}

// The slot's feeding warp, in step, one elected lane issuing.
static __device__ __noinline__ void fa_feed(uint32_t s) {
  FaShared *S = fa_shared();
  const FaTask &F = *fa_task();
  volatile uint32_t *failed = &S->failed;
  const unsigned long long budget = F.budget;
  const DTmap *tm = F.tm_q;
  const uint32_t lane = threadIdx.x & 31u, q_s = F.base + s * kFaQ, k_s = F.base + kFaSlots * kFaQ + s * kFaStages * kFaKv;
  const uint32_t v_s = k_s + kFaSlots * kFaStages * kFaKv;
  const uint32_t tmem = S->tmem_base + s * kFaSlotCols;
  const bool k_mn = F.k_mn != 0u;
  const uint32_t fmt = F.adt == kBF16 ? 1u : 0u;
  // S: A = Q (K-major), B = K block; O: A = P (tensor memory), B = V (d is the unit-stride "MN" dimension)
  const uint32_t idesc_s = (1u << 4) | (fmt << 7) | (fmt << 10) | ((k_mn ? 1u : 0u) << 16) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
  const uint32_t idesc_o = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
  // descriptors of stage 0; the others differ in the 16-byte-unit address field only
  const uint64_t dq = tc_desc(q_s, 16u, 1024u), dk = k_mn ? tc_desc(k_s, 8192u, 1024u) : tc_desc(k_s, 16u, 1024u), dv = tc_desc(v_s, 8192u, 1024u);
  const uint64_t adv_k = k_mn ? (2048u >> 4) : (32u >> 4);
  fence_proxy_async_global();          // operands written by the previous phase's ordinary stores
  __syncwarp();
  const bool leader = elect_one_sync();
  uint32_t u_next = F.first + s;                                        // static
  uint32_t first_draw = F.stop ? F.first + s * (F.stop / kFaSlots) : kFaNone;      // dynamic
  auto next = [&]() -> uint32_t {      // tiles that see no key have no result
    for (;;) {
      uint32_t u;
      if (F.work) {
        // A slot's first tile is its own, so that few tiles go to one slot of each lane (all three of the lanes that come first drew
        // them: 252 tiles of up to 777 keys 32 us, 25 so); the counter gives out what is left.
        uint32_t tk = first_draw;
        if (tk == kFaNone) {
          if (lane == 0u) tk = atomicAdd(F.work, 1u);
          tk = __shfl_sync(0xffffffffu, tk, 0) + F.stop;
        }
        first_draw = kFaNone;
        if (tk >= static_cast<uint32_t>(F.H) * static_cast<uint32_t>(F.per_head)) return kFaNone;
        // heaviest first: with a causal mask the last rows of a head see the most keys
        const uint32_t lvl = tk / static_cast<uint32_t>(F.H), g = tk - lvl * static_cast<uint32_t>(F.H);
        u = g * static_cast<uint32_t>(F.per_head) + (F.causal ? static_cast<uint32_t>(F.per_head) - 1u - lvl : lvl);
      } else {
        if (u_next >= F.stop) return kFaNone;
        u = u_next;
        u_next += kFaSlots;
      }
      if (fa_tile(F, u).blocks > 0) return u;
    }
  };
  struct Place { int32_t m0, h0, h1, blocks; };
  auto place = [&](uint32_t u) {
    const FaTile t = fa_tile(F, u);
    const int32_t h1 = t.g / static_cast<int32_t>(F.h0_size);
    return Place{t.m0, t.g - h1 * static_cast<int32_t>(F.h0_size), h1, t.blocks};
  };
  auto load_q = [&](const Place &t) {
    if (leader) {
      mbar_arrive_tx(&S->q_full[s], kFaQ);
      tma_load_4d(q_s, tm, 0, t.m0, t.h0, t.h1, &S->q_full[s]);                        // rows past T arrive as zeros
    }
  };
  // block j of the tile, number blk of all
  auto load_k = [&](const Place &t, int32_t j, uint32_t blk) {
    const uint32_t st = blk % kFaStages, dst = k_s + st * kFaKv;
    if (leader && j < t.blocks) {
      mbar_arrive_tx(&S->k_full[s][st], kFaKv);
      if (k_mn) tma_load_4d(dst, tm + 1, j * 64, 0, t.h0, t.h1, &S->k_full[s][st]);    // K as [d][keys]
      else tma_load_4d(dst, tm + 1, 0, j * 64, t.h0, t.h1, &S->k_full[s][st]);
    }
  };
  auto load_v = [&](const Place &t, int32_t j, uint32_t blk) {
    const uint32_t st = blk % kFaStages;
    if (leader && j < t.blocks) {
      mbar_arrive_tx(&S->v_full[s][st], kFaKv);
      tma_load_4d(v_s + st * kFaKv, tm + 2, 0, j * 64, t.h0, t.h1, &S->v_full[s][st]);
    }
  };
  auto post = [&](uint32_t u, uint32_t n) {
    if (leader) {
      S->tile[s][n & 1u] = u;
      mbar_arrive(&S->t_full[s]);
    }
    __syncwarp();
  };
  uint32_t n = 0, b = 0;               // tiles and key blocks so far
  bool ok = true;
  uint32_t u = next();
  post(u, n);
  if (u == kFaNone) return;
  Place t = place(u);
  load_q(t);
  for (uint32_t j = 0; j < kFaStages; ++j) { load_k(t, static_cast<int32_t>(j), j); if (j < 2u) load_v(t, static_cast<int32_t>(j), j); }
  for (;;) {
    u = next();                        // (its atomic under the loads' flight)
    ok = tc_wait_uniform(&S->q_full[s], n & 1u, failed, budget);
    // O (+)= P V of block `blk`, number j of the tile
    auto product = [&](int32_t j, uint32_t blk) {
      const uint32_t st = blk % kFaStages;
      ok = ok && tc_wait_uniform(&S->v_full[s][st], (blk / kFaStages) & 1u, failed, budget) && tc_wait_uniform(&S->p_full[s], blk & 1u, failed, budget);
      if (!ok) return;
      tc_fence_after_sync();
      const uint64_t db = dv + ((st * kFaKv) >> 4);
      if (leader) {
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) tc_mma_f16_ts(tmem + 64u, tmem + 128u + 8u * k, db + k * (2048u >> 4), idesc_o, (j > 0 || k > 0u) ? 1u : 0u);
        tc_commit(&S->pv_done[s]);
      }
      __syncwarp();
      // P(j) is full: the softmax saw the product before this one done
      load_v(t, j + 2, blk + 2u);
    };
    for (int32_t j = 0; ok && j < t.blocks; ++j, ++b) {
      const uint32_t st = b % kFaStages;
      ok = tc_wait_uniform(&S->k_full[s][st], (b / kFaStages) & 1u, failed, budget) && (b == 0u || tc_wait_uniform(&S->s_free[s], (b - 1u) & 1u, failed, budget));
      if (!ok) break;
      tc_fence_after_sync();
      const uint64_t db = dk + ((st * kFaKv) >> 4);
      if (leader) {
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) tc_mma_f16(tmem, dq + k * (32u >> 4), db + k * adv_k, idesc_s, k ? 1u : 0u);
        tc_commit(&S->s_full[s]);
      }
      __syncwarp();
      if (j > 0) {
        load_k(t, j + 2, b + 2u);      // the scores before have been read, so their product is done
        product(j - 1, b - 1u);
      }
    }
    // The last scores are read: Q and all stages of K are free for the next tile, V's but for the last two blocks'.
    ok = ok && tc_wait_uniform(&S->s_free[s], (b - 1u) & 1u, failed, budget);
    if (!ok) return;
    post(u, ++n);
    Place t2 = t;
    if (u != kFaNone) {
      t2 = place(u);
      load_q(t2);
      for (uint32_t j = 0; j < kFaStages; ++j) load_k(t2, static_cast<int32_t>(j), b + j);
      load_v(t2, 0, b);
    }
    product(t.blocks - 1, b - 1u);
    if (!ok) return;
    if (u == kFaNone) {
      if (lane == 0u) tc_drain(&S->pv_done[s], 1u, b, failed, budget);
      __syncwarp();
      return;
    }
    load_v(t2, 1, b + 1u);
    t = t2;
  }
}

// One of the slot's softmax warps: rows 32 q4 .. + 31 of its tiles, a thread each.
template <bool BF>
static __device__ __noinline__ void fa_rows(uint32_t s, uint32_t q4) {
  FaShared *S = fa_shared();
  const FaTask &F = *fa_task();
  volatile uint32_t *failed = &S->failed;
  const unsigned long long budget = F.budget;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t s_addr = S->tmem_base + ((32u * q4) << 16) + s * kFaSlotCols, o_addr = s_addr + 64u, p_addr = s_addr + 128u;
  const float sl2 = F.sl2;
  const unsigned long long sl2_2 = pack_f32x2(sl2, sl2);
  uint32_t n = 0, b = 0;
  for (;; ++n) {
    if (!tc_wait_uniform(&S->t_full[s], n & 1u, failed, budget)) return;
    const uint32_t u = *reinterpret_cast<volatile uint32_t *>(&S->tile[s][n & 1u]);
    if (u == kFaNone) return;
    const FaTile t = fa_tile(F, u);
    const int32_t m = t.m0 + static_cast<int32_t>(32u * q4 + lane);
    const int32_t c_end = F.causal ? min(F.C, m + (F.C - F.T) + 1) : F.C;      // keys this row may see
    float m_used = -INFINITY, l_run = 0.0f;
#pragma unroll 1
    for (int32_t j = 0; j < t.blocks; ++j, ++b) {
      if (!tc_wait_uniform(&S->s_full[s], b & 1u, failed, budget)) return;
      tc_fence_after_sync();
      uint32_t lo[32], hi[32];
      __syncwarp();
      tc_ld32(s_addr, lo);
      tc_ld32(s_addr + 32u, hi);
      tc_wait_ld();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0u) mbar_arrive(&S->s_free[s]);          // the scores are in registers: the slot's next may be written
      const int32_t lim = c_end - j * 64;
      if (lim < 64) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i >= lim) lo[i] = 0xff800000u;               // -inf
          if (i + 32 >= lim) hi[i] = 0xff800000u;
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};     // four independent chains
#pragma unroll
      for (int i = 0; i < 32; ++i) mx4[i & 3] = max3(mx4[i & 3], __uint_as_float(lo[i]), __uint_as_float(hi[i]));
      // sl2 > 0 for every softmax scale in use; a non-positive scale takes the CUDA-core path
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
      // the maximum in use moves only when the row's true maximum outgrew it by 2^8
      const bool grow = mx > m_used + kFaRescale;
      bool waited = j == 0;                                // (at a tile's start the product before was waited for, for the result)
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = !grow ? 1.0f : (m_used == -INFINITY ? 0.0f : fast_ex2(m_used - mx));
        if (j > 0) {
          if (!tc_wait_uniform(&S->pv_done[s], (b - 1u) & 1u, failed, budget)) return;
          tc_fence_after_sync();
          waited = true;
#pragma unroll 1
          for (uint32_t cb = 0; cb < 64u; cb += 16u) {
            uint32_t raw[16];
            __syncwarp();
            tc_ld16(o_addr + cb, raw);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) raw[i] = __float_as_uint(__uint_as_float(raw[i]) * alpha);
            tc_st16(o_addr + cb, raw);
          }
          tc_wait_st();
        }
        if (grow) { l_run *= alpha; m_used = mx; }
      }
      const float neg_m = m_used == -INFINITY ? 0.0f : -m_used;
      const unsigned long long neg_2 = pack_f32x2(neg_m, neg_m);
      // p = 2^(s - m_used), two to a 32-bit column
      uint32_t pk[32];
      unsigned long long sum[2] = {0ull, 0ull};
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float s0 = __uint_as_float(i < 16 ? lo[2 * i] : hi[2 * i - 32]), s1 = __uint_as_float(i < 16 ? lo[2 * i + 1] : hi[2 * i - 31]);
        float e0, e1;
        unpack_f32x2(fma_f32x2(pack_f32x2(s0, s1), sl2_2, neg_2), e0, e1);
        e0 = fast_ex2(e0);
        e1 = fast_ex2(e1);
        pk[i] = BF ? cvt_bf16x2(e1, e0) : cvt_f16x2(e1, e0);
        sum[i & 1] = add_f32x2(sum[i & 1], pack_f32x2(e0, e1));
      }
      float a0, a1;
      unpack_f32x2(add_f32x2(sum[0], sum[1]), a0, a1);
      l_run += a0 + a1;
      // P's columns are free when the product before has read them
      if (!waited && !tc_wait_uniform(&S->pv_done[s], (b - 1u) & 1u, failed, budget)) return;
      tc_fence_after_sync();
      __syncwarp();
      tc_st32(p_addr, pk);
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0u) mbar_arrive(&S->p_full[s]);
    }
    // ---- output: O / l ----
    if (!tc_wait_uniform(&S->pv_done[s], (b - 1u) & 1u, failed, budget)) return;
    tc_fence_after_sync();
    const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
#pragma unroll 1
    for (uint32_t cb = 0; cb < 64u; cb += 32u) {
      uint32_t raw[32];
      __syncwarp();
      tc_ld32(o_addr + cb, raw);
      tc_wait_ld();
      if (m < F.T) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(raw[i]) * inv;
        tc_store_row32(F.out, F.dt, (static_cast<int64_t>(t.g) * F.T + m) * 64 + cb, v, 32, true);
      }
    }
    tc_fence_before_sync();
  }
}

template <typename Lane>
static __device__ __noinline__ bool flash_tc_tiles(const Lane &L, const DTask &t, uint32_t tile_lo, uint32_t tile_hi) {
  const KParams &P = *L.P;
  const DFlash &df = *reinterpret_cast<const DFlash *>(P.desc + t.desc);
  const int32_t *x = P.aux + t.p[3];
  const int64_t H = x[0], T = x[1];
  uint8_t *out = resolve(P, t.ptr[0]);
  if (df.tmap < 0 || (reinterpret_cast<uintptr_t>(out) & 15u)) return false;
  const bool dynamic = df.work_slot != kNoWorkSlot;
  const int64_t rows_end = min(static_cast<int64_t>(tile_hi), H * T);
  if (static_cast<int64_t>(tile_lo) >= rows_end && !dynamic) return true;

  B2_DYN_SMEM(sm);
  FaShared *S = fa_shared();
  FaTask *F = fa_task();
  const uint32_t w = __shfl_sync(0xffffffffu, L.tid / kWarp, 0);   // the warp index, provably uniform
  __syncthreads();   // the scratch slot and the workspace are free
  if (L.tid == 0) {
    for (uint32_t s = 0; s < kFaSlots; ++s) {
      mbar_init(&S->t_full[s], 1); mbar_init(&S->q_full[s], 1);
      for (uint32_t k = 0; k < kFaStages; ++k) { mbar_init(&S->k_full[s][k], 1); mbar_init(&S->v_full[s][k], 1); }
      mbar_init(&S->s_full[s], 1); mbar_init(&S->s_free[s], 4); mbar_init(&S->p_full[s], 4); mbar_init(&S->pv_done[s], 1);
    }
    S->failed = 0u;
    const int64_t per_head = (T + 127) / 128;
    // static mode: the tiles whose first row lies in [tile_lo, rows_end)
    auto tile_at_or_after = [&](int64_t row) {
      const int64_t g = row / T, m = row % T;
      return static_cast<uint32_t>(g * per_head + (m + 127) / 128);
    };
    F->tm_q = P.tmaps + df.tmap;
    F->work = dynamic ? reinterpret_cast<RedScratch *>(P.scratch)->work + 2u * df.work_slot : nullptr;
    F->out = out;
    F->budget = P.wait_budget_ns;
    F->H = x[0]; F->T = x[1]; F->C = x[2]; F->per_head = static_cast<int32_t>(per_head);
    const bool all_lanes = df.n_owner_lanes == P.n_lanes;             // (a lane's number is its number among the owners)
    F->first = dynamic ? L.lane : tile_at_or_after(static_cast<int64_t>(tile_lo));
    F->stop = dynamic ? (all_lanes ? kFaSlots * P.n_lanes : 0u) : tile_at_or_after(rows_end);
    F->h0_size = df.h0_size; F->causal = x[5] != 0 ? 1u : 0u; F->k_mn = df.k_mn; F->adt = t.adt; F->dt = t.dt;
    F->base = (smem_addr(sm + kSmemSys) + 1023u) & ~1023u;
    F->sl2 = __int_as_float(x[4]) * 1.4426950408889634f;   // scores in the log2 domain
    fence_mbar_init();
  }
  if (w == 3u) {
    __syncwarp();
    tmem_alloc(&S->tmem_base, kFaCols);
  }
  fence_proxy_async_smem();   // what the entry before wrote here by ordinary stores, before asynchronous copies overwrite it
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (w < kFaSlots) fa_feed(w);
  else if (w >= 4u) {
    if (t.adt == kBF16) fa_rows<true>((w - 4u) >> 2, w & 3u);
    else fa_rows<false>((w - 4u) >> 2, w & 3u);
  }

  // ---------------- teardown ----------------
  // (no copy or product is under way: the feeding warps waited for the last products, the products for every copy)
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  const bool gave_up = S->failed != 0u;
  if (gave_up) {     // copies / matmuls of other roles may still be landing: give them time (see ops_mma_tc.cuh)
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) nanosleep_ns(1000);
  }
  if (w == 3u) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(S->tmem_base, kFaCols);
  }
  if (L.tid == 0) {
    if (gave_up) {
      set_status(P, kStTensorTimeout, L.lane, tile_lo, kTopFlashAttn);
    } else {
      for (uint32_t s = 0; s < kFaSlots; ++s) {
        mbar_inval(&S->t_full[s]); mbar_inval(&S->q_full[s]);
        for (uint32_t k = 0; k < kFaStages; ++k) { mbar_inval(&S->k_full[s][k]); mbar_inval(&S->v_full[s][k]); }
        mbar_inval(&S->s_full[s]); mbar_inval(&S->s_free[s]); mbar_inval(&S->p_full[s]); mbar_inval(&S->pv_done[s]);
      }
    }
    if (dynamic) {
      // the last lane to finish puts the counters back to rest for the task's next run
      uint32_t *work = F->work;
      __threadfence();
      if (atomicAdd(&work[1], 1u) == df.n_owner_lanes - 1u) { st_relaxed_gpu(&work[0], 0u); st_relaxed_gpu(&work[1], 0u); }
    }
  }
  __syncthreads();
  return true;
}

#else

__device__ __forceinline__ bool flash_tc_tiles(const Lane &, const DTask &, uint32_t, uint32_t) { return false; }

#endif

}  // namespace b2
#endif
