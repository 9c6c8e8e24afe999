// The common row pipelines of kTopFuseRows as straight-line code: an optional residual sum (stored on the way), LayerNorm
// or RMS norm, x gamma, + beta, GELU, softmax, an optional full sum, store - each stage there or not by a flag that is
// uniform over the task. The step interpreter (ops_fuse.cuh) runs the same rows at ~85 instructions per element: at every
// step's join the compiler moves a thread's elements between registers; here they stay where they are (~35).
// LayerNorm, gamma, beta, GELU, softmax, sum on 8192 x 4096: f32 186 -> 96 us, bf16 189 -> 103 us; 3001 x 1000 in
// bf16 148 -> 23 us ("before": the tile ops one after another, barriers between rows of other lengths than 4096).
#ifndef B2VM_OPS_ROWPIPE_CUH_
#define B2VM_OPS_ROWPIPE_CUH_

#include "ops_fuse.cuh"

namespace b2 {

struct RowPipe {            // resolved, in shared memory
  uint32_t flags, cols, n_buf, stage_off, mul_off, add_off;   // n_buf: row buffers per thread, 2 or 4; *_off: staged vectors (byte offset), kFuNoSlot = read from memory
  float eps, s, t;
  uint32_t pad;
  const uint8_t *x, *y, *mul, *add;
  uint8_t *mid, *out;       // the stored residual sum; the result
};
constexpr uint32_t kPipeArgs = kSmemChain;      // the elementwise chain cache's place
static_assert(sizeof(RowPipe) <= 512, "fits there");

template <int DT>
__device__ __forceinline__ float pipe_q(float v) {
  if (DT == kBF16) return __uint_as_float(cvt_bf16x2(v, 0.0f) & 0xffff0000u);
  if (DT == kF16) return f16_bits_to_f32(f32_to_f16_bits(v));
  return v;
}
// four values rounded to the storage type, two conversions for bf16
template <int DT>
__device__ __forceinline__ void pipe_q4(float (&v)[4]) {
  if (DT == kBF16) {
    const uint32_t a = cvt_bf16x2(v[1], v[0]), b = cvt_bf16x2(v[3], v[2]);
    v[0] = __uint_as_float(a << 16); v[1] = __uint_as_float(a & 0xffff0000u);
    v[2] = __uint_as_float(b << 16); v[3] = __uint_as_float(b & 0xffff0000u);
  } else if (DT == kF16) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = pipe_q<DT>(v[e]);
  }
}
template <int DT>
__device__ __forceinline__ void pipe_ld4(const uint8_t *p, float (&v)[4]) {
  if (DT == kF32) {
    const float4 f = *reinterpret_cast<const float4 *>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const uint2 w = *reinterpret_cast<const uint2 *>(p);
    if (DT == kBF16) {
      v[0] = __uint_as_float(w.x << 16); v[1] = __uint_as_float(w.x & 0xffff0000u);
      v[2] = __uint_as_float(w.y << 16); v[3] = __uint_as_float(w.y & 0xffff0000u);
    } else {
      v[0] = f16_bits_to_f32(w.x & 0xffffu); v[1] = f16_bits_to_f32(w.x >> 16);
      v[2] = f16_bits_to_f32(w.y & 0xffffu); v[3] = f16_bits_to_f32(w.y >> 16);
    }
  }
}
template <int DT>
__device__ __forceinline__ void pipe_st4(uint8_t *p, const float (&v)[4]) {
  if (DT == kF32) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if (DT == kBF16) *reinterpret_cast<uint2 *>(p) = make_uint2(cvt_bf16x2(v[1], v[0]), cvt_bf16x2(v[3], v[2]));
  else *reinterpret_cast<uint2 *>(p) = make_uint2(f32_to_f16_bits(v[0]) | (f32_to_f16_bits(v[1]) << 16), f32_to_f16_bits(v[2]) | (f32_to_f16_bits(v[3]) << 16));
}
template <int DT>
__device__ __forceinline__ float pipe_ld1(const uint8_t *p, uint32_t i) {
  if (DT == kF32) return reinterpret_cast<const float *>(p)[i];
  const uint32_t h = reinterpret_cast<const uint16_t *>(p)[i];
  return DT == kBF16 ? __uint_as_float(h << 16) : f16_bits_to_f32(h);
}
template <int DT>
__device__ __forceinline__ void pipe_st1(uint8_t *p, uint32_t i, float v) {
  if (DT == kF32) reinterpret_cast<float *>(p)[i] = v;
  else if (DT == kBF16) reinterpret_cast<uint16_t *>(p)[i] = static_cast<uint16_t>(cvt_bf16x2(0.0f, v));
  else reinterpret_cast<uint16_t *>(p)[i] = static_cast<uint16_t>(f32_to_f16_bits(v));
}

template <int DT, int G, bool VEC>
static __device__ __noinline__ float row_pipe_run(uint32_t tid, uint32_t nthr, uint32_t T, uint32_t lo, uint32_t hi) {
  B2_DYN_SMEM(sm);
  const RowPipe &A = *reinterpret_cast<const RowPipe *>(sm + kPipeArgs);
  constexpr uint32_t ESZ = DT == kF32 ? 4u : 2u;
  const uint32_t gi = tid / T, gl = tid % T, ng = nthr / T, cols = A.cols, fl = A.flags;
  float *slot = reinterpret_cast<float *>(sm + kFuseSlots) + (T > 32u ? gi * 64u : 0u);
  uint32_t turn = 0;
  const uint32_t nv = VEC ? (cols > gl * 4u ? (cols - gl * 4u + 4u * T - 1u) / (4u * T) : 0u) : (cols > gl ? (cols - gl + T - 1u) / T : 0u);
  const uint32_t c0 = VEC ? gl * 4u : gl, cstep = VEC ? 4u * T : T;      // column of (group 0 | element 0), and from one to the next
  const float inv_n = 1.0f / static_cast<float>(cols);
  // staging of the rows ahead: [n_buf][x, y][G][threads] words of 4 elements
  constexpr uint32_t W = 4u * ESZ;
  const uint32_t nsrc = (fl & kRpRes) ? 2u : 1u;
  uint8_t *stage = sm + A.stage_off + tid * W;
  const uint32_t gstride = nthr * W, bufstride = nsrc * G * gstride;
  auto start = [&](uint32_t row, uint32_t buf) {
    const size_t off = (static_cast<size_t>(row) * cols + c0) * ESZ;
    if (VEC) {
      uint32_t d = smem_addr(stage) + buf * bufstride;
#pragma unroll 1
      for (uint32_t k = 0; k < nsrc; ++k) {
        const uint8_t *q = (k ? A.y : A.x) + off;
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if (static_cast<uint32_t>(g) < nv) {
            if (ESZ == 4u) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + g * gstride), "l"(q + g * (cstep * ESZ)) : "memory");
            else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d + g * gstride), "l"(q + g * (cstep * ESZ)) : "memory");
          }
        }
        d += G * gstride;
      }
    } else {
      const uint8_t *q = A.x + static_cast<size_t>(row) * cols * ESZ;
      for (uint32_t b = gl * 128u; b < cols * ESZ; b += T * 128u) prefetch_l2(q + b);
      if (fl & kRpRes) {
        q = A.y + static_cast<size_t>(row) * cols * ESZ;
        for (uint32_t b = gl * 128u; b < cols * ESZ; b += T * 128u) prefetch_l2(q + b);
      }
    }
  };
#define B2_RP_G _Pragma("unroll") for (int g = 0; g < G; ++g)
#define B2_RP_E _Pragma("unroll") for (int e = 0; e < 4; ++e)
#define B2_RP_IN(g, e) (static_cast<uint32_t>(VEC ? (g) : 4 * (g) + (e)) < nv)
  auto add_f = [](float a, float c) { return a + c; };
  float csum = 0.0f;
  const uint32_t ahead = VEC ? A.n_buf - 1u : 1u;       // rows under way beyond the current one (one commit group per row)
  uint32_t buf = 0, row = lo + gi;
  for (uint32_t k = 0; k < ahead; ++k) {
    if (row + k * ng < hi) start(row + k * ng, k);
    cp_async_commit();
  }
  for (; row < hi; row += ng) {
    float X[G][4];
    if (VEC) {
      if (ahead == 3u) cp_async_wait<2>(); else cp_async_wait<0>();
    }
    if (row + ahead * ng < hi) start(row + ahead * ng, VEC ? (buf + ahead) & ahead : 0u);
    cp_async_commit();
    const size_t base = static_cast<size_t>(row) * cols * ESZ;
    // a second operand over the row: staged, or straight from memory
    auto dense = [&](const uint8_t *p, uint32_t k, int g, float (&v)[4]) {
      if (VEC) {
        if (static_cast<uint32_t>(g) < nv) pipe_ld4<DT>(stage + buf * bufstride + (k * G + g) * gstride, v);
        else v[0] = v[1] = v[2] = v[3] = 0.0f;
      } else {
        B2_RP_E v[e] = B2_RP_IN(g, e) ? pipe_ld1<DT>(p + base, c0 + (4 * g + e) * cstep) : 0.0f;
      }
    };
    auto column = [&](const uint8_t *p, uint32_t off, int g, float (&v)[4]) {
      const uint8_t *q = off != kFuNoSlot ? sm + off : p;
      if (VEC) {
        if (static_cast<uint32_t>(g) < nv) pipe_ld4<DT>(q + (c0 + g * cstep) * ESZ, v);
        else v[0] = v[1] = v[2] = v[3] = 0.0f;
      } else {
        B2_RP_E v[e] = B2_RP_IN(g, e) ? pipe_ld1<DT>(q, c0 + (4 * g + e) * cstep) : 0.0f;
      }
    };
    auto store = [&](uint8_t *p) {
      B2_RP_G {
        if (VEC) {
          if (static_cast<uint32_t>(g) < nv) pipe_st4<DT>(p + base + (c0 + g * cstep) * ESZ, X[g]);
        } else {
          B2_RP_E if (B2_RP_IN(g, e)) pipe_st1<DT>(p + base, c0 + (4 * g + e) * cstep, X[g][e]);
        }
      }
    };
    B2_RP_G dense(A.x, 0u, g, X[g]);
    if (fl & kRpRes) {
      B2_RP_G {
        float Y[4];
        dense(A.y, 1u, g, Y);
        B2_RP_E X[g][e] = __fadd_rn(X[g][e], Y[e]);
        pipe_q4<DT>(X[g]);
      }
      if (A.mid) store(A.mid);
    }
    if (fl & kRpLn) {
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f}, b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      B2_RP_G B2_RP_E { a[e] += X[g][e]; b[e] = fmaf(X[g][e], X[g][e], b[e]); }         // zeros past the row's end
      const float2 r = fuse_group_reduce2((a[0] + a[1]) + (a[2] + a[3]), (b[0] + b[1]) + (b[2] + b[3]), add_f, slot, T, gi, gl, turn);
      const float mu = r.x * inv_n, var = __fsub_rn(r.y * inv_n, __fmul_rn(mu, mu)), rden = rsqrt_nr(__fadd_rn(var, A.eps));
      B2_RP_G { B2_RP_E X[g][e] = (X[g][e] - mu) * rden; if (fl & kRpQ) pipe_q4<DT>(X[g]); }
    } else if (fl & kRpRms) {
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      B2_RP_G B2_RP_E a[e] = __fadd_rn(a[e], __fmul_rn(X[g][e], X[g][e]));
      const float ss = fuse_group_reduce((a[0] + a[1]) + (a[2] + a[3]), add_f, slot, T, gi, gl, turn);
      const float r = rsqrt_nr_tiny(affine2(ss, A.s, A.t));
      B2_RP_G { B2_RP_E X[g][e] = __fmul_rn(X[g][e], r); if (fl & kRpQ) pipe_q4<DT>(X[g]); }
    }
    if (fl & kRpMul) {
      B2_RP_G {
        float Y[4];
        column(A.mul, A.mul_off, g, Y);
        B2_RP_E X[g][e] = __fmul_rn(X[g][e], Y[e]);
        if (fl & kRpQ) pipe_q4<DT>(X[g]);
      }
    }
    if (fl & kRpAdd) {
      B2_RP_G {
        float Y[4];
        column(A.add, A.add_off, g, Y);
        B2_RP_E X[g][e] = __fadd_rn(X[g][e], Y[e]);
        if (fl & kRpQ) pipe_q4<DT>(X[g]);
      }
    }
    if (fl & kRpGelu) {
      B2_RP_G { B2_RP_E X[g][e] = gelu_tanh(X[g][e]); if (fl & kRpQ) pipe_q4<DT>(X[g]); }
    }
    if (fl & kRpSoftmax) {
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      B2_RP_G B2_RP_E if (B2_RP_IN(g, e)) m4[e] = fmaxf(m4[e], X[g][e]);               // a NaN still poisons the row through the sum
      const float m = fuse_group_reduce(fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])), [](float a, float c) { return fmaxf(a, c); }, slot, T, gi,
                                        gl, turn);
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      B2_RP_G B2_RP_E {
        X[g][e] = fast_ex2((X[g][e] - m) * 1.4426950408889634f);
        if (B2_RP_IN(g, e)) a[e] += X[g][e];
      }
      const float s = fuse_group_reduce((a[0] + a[1]) + (a[2] + a[3]), add_f, slot, T, gi, gl, turn);
      const float rs = rcp_nr(s);
      B2_RP_G { B2_RP_E X[g][e] *= rs; if (fl & kRpQ) pipe_q4<DT>(X[g]); }
    }
    if (DT != kF32 && !(fl & kRpQ)) B2_RP_G pipe_q4<DT>(X[g]);
    if (fl & kRpCarry) {
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      B2_RP_G B2_RP_E if (B2_RP_IN(g, e)) a[e] += X[g][e];
      csum += (a[0] + a[1]) + (a[2] + a[3]);
    }
    if (A.out) store(A.out);
    if (VEC) buf = (buf + 1u) & ahead;
  }
#undef B2_RP_IN
#undef B2_RP_E
#undef B2_RP_G
  cp_async_wait_all();
  return csum;
}

// RMS norm x gamma of 16-bit rows up to 1024 columns, a warp per row: 16-byte loads straight into registers, the next row's under
// this one's arithmetic. Bound: HBM. The general pipeline spends ~60 instructions an element on its staging and optional stages and
// took 34 us for 16384 x 1024 (67 MB); this is about 6.
template <int DT>
static __device__ __noinline__ void rms_rows(const Lane &L, const DPipe &p, uint32_t cols, uint32_t lo, uint32_t hi) {
  const KParams &P = *L.P;
  const uint8_t *x = resolve(P, p.x), *gam = resolve(P, p.mul);
  uint8_t *out = resolve(P, p.out);
  const uint32_t w = L.tid / kWarp, l = L.tid % kWarp, nw = L.nthr / kWarp, words = cols / 8u;
  uint4 *gs = reinterpret_cast<uint4 *>(L.smem + kFuseData);
  for (uint32_t i = L.tid; i < words; i += L.nthr) gs[i] = ldg_v4(gam + 16u * i);
  __syncthreads();
  uint4 v[4], n[4];
  auto load = [&](uint32_t row) {
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
      n[k] = row < hi && l + 32u * k < words ? ldg_v4(x + (static_cast<size_t>(row) * words + l + 32u * k) * 16u) : make_uint4(0u, 0u, 0u, 0u);
  };
  load(lo + w);
#pragma unroll 1
  for (uint32_t row = lo + w; row < hi; row += nw) {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = n[k];
    load(row + nw);
    float ss[2] = {0.0f, 0.0f}, f[8], g[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      unpack8(v[k], DT, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) ss[e & 1] = fmaf(f[e], f[e], ss[e & 1]);
    }
    const float r = rsqrt_nr_tiny(affine2(warp_reduce(ss[0] + ss[1], [](float a, float c) { return a + c; }), p.s, p.t));
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
      if (l + 32u * k < words) {
        unpack8(v[k], DT, f);
        unpack8(gs[l + 32u * k], DT, g);
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float a = __fmul_rn(__fmul_rn(f[2 * i], r), g[2 * i]), b = __fmul_rn(__fmul_rn(f[2 * i + 1], r), g[2 * i + 1]);
          o[i] = DT == kBF16 ? cvt_bf16x2(b, a) : (f32_to_f16_bits(a) | (f32_to_f16_bits(b) << 16));
        }
        stg_v4(out + (static_cast<size_t>(row) * words + l + 32u * k) * 16u, make_uint4(o[0], o[1], o[2], o[3]));
      }
    }
  }
  __syncthreads();
}

// All threads. The task's shared descriptor `f` names a pipeline (f.pipe != 0).
static __device__ __noinline__ void row_pipe_tiles(const Lane &L, const DTask &t, const DFuse &f, uint32_t tile_lo, uint32_t tile_hi) {
  const KParams &P = *L.P;
  const DPipe &p = f.pipe;
  RowPipe *A = reinterpret_cast<RowPipe *>(L.smem + kPipeArgs);
  const uint32_t cols = f.cols, hi = min(tile_hi, f.rows), esz = dt_size(p.dt);
  // (fewer rows than warps: several warps per row, below, are sooner done)
  if (p.flags == (kRpOn | kRpRms | kRpMul) && p.dt != kF32 && p.out && !p.mid && f.vec && cols % 8u == 0u && cols <= 1024u && hi >= tile_lo + 16u) {
    if (p.dt == kBF16) rms_rows<kBF16>(L, p, cols, tile_lo, hi);
    else rms_rows<kF16>(L, p, cols, tile_lo, hi);
    return;
  }
  const PipeShape sh = pipe_shape(p.flags, esz, f.vec != 0u, cols, hi - tile_lo, L.nthr);
  const uint32_t T = sh.T, G = sh.G, buf_bytes = sh.buf_bytes, stage_bytes = 2u * buf_bytes;      // (two buffers fit: the loader saw to it)
  const uint32_t vbytes = (cols * esz + 15u) & ~15u;
  const uint32_t nvec = ((p.flags & kRpMul) ? 1u : 0u) + ((p.flags & kRpAdd) ? 1u : 0u);
  const bool keep = hi - tile_lo > 1u && kFuseData + nvec * vbytes + stage_bytes <= L.smem_bytes;     // column vectors in shared memory
  const uint8_t *mul = p.mul ? resolve(P, p.mul) : nullptr, *add = p.add ? resolve(P, p.add) : nullptr;
  uint32_t off = kFuseData;
  uint32_t offs[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint8_t *src = k ? add : mul;
    offs[k] = kFuNoSlot;
    if (!src || !keep) continue;
    offs[k] = off;
    const uint32_t words = cols * esz / 4u;
    for (uint32_t i = L.tid; i < words; i += L.nthr) reinterpret_cast<uint32_t *>(L.smem + off)[i] = ldg_u32(src + 4u * i);
    if (L.tid == 0 && (cols * esz) % 4u) *reinterpret_cast<uint16_t *>(L.smem + off + 4u * words) = static_cast<uint16_t>(ldg_u16(src + 4u * words));
    off += vbytes;
  }
  if (L.tid == 0) {
    A->flags = p.flags; A->cols = cols; A->n_buf = ((off + 15u) & ~15u) + 4u * buf_bytes <= L.smem_bytes ? 4u : 2u; A->stage_off = (off + 15u) & ~15u; A->mul_off = offs[0]; A->add_off = offs[1];
    A->eps = p.eps; A->s = p.s; A->t = p.t;
    A->x = resolve(P, p.x); A->y = p.y ? resolve(P, p.y) : nullptr;
    A->mul = mul; A->add = add;
    A->mid = p.mid ? resolve(P, p.mid) : nullptr;
    A->out = p.out ? resolve(P, p.out) : nullptr;
  }
  __syncthreads();
  float csum = 0.0f;
  if (tile_lo < hi) {
#define B2_RP3(D, GG) (f.vec ? row_pipe_run<D, GG, true>(L.tid, L.nthr, T, tile_lo, hi) : row_pipe_run<D, GG, false>(L.tid, L.nthr, T, tile_lo, hi))
#define B2_RP2(D) (G == 1u ? B2_RP3(D, 1) : G == 2u ? B2_RP3(D, 2) : G == 4u ? B2_RP3(D, 4) : B2_RP3(D, 8))
    csum = p.dt == kF32 ? B2_RP2(kF32) : p.dt == kBF16 ? B2_RP2(kBF16) : B2_RP2(kF16);
#undef B2_RP2
#undef B2_RP3
  }
  if (f.total) fuse_full_sum(L, csum, reinterpret_cast<float *>(resolve(P, f.total)), t.p[3], f.n_owner_lanes);
}

}  // namespace b2
#endif
