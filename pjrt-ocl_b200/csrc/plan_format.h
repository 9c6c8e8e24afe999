// Descriptors of the re-planner's own ops (replan.h), shared by the loader and plan_kernel.cu.
#ifndef B2VM_PLAN_FORMAT_H_
#define B2VM_PLAN_FORMAT_H_

#include "format.h"

namespace b2 {

// ---- steps of a fused op ---------------------------------------------------------------
//
// A fused op carries one value X per element through a list of steps; Y holds a second operand. Values are f32
// in registers whatever the storage type (bf16 and f16 are exact in f32; kFuQuant rounds to the type a value
// would have been stored with). The same list format drives the row pipelines and the matmul epilogues.
enum FuCode : uint32_t {
  kFuLoadX = 0, kFuLoadY,          // dense operand (the op's own element index)
  kFuRowVecY,                      // one value per column
  kFuColVecY,                      // one value per row
  kFuScalarY,                      // one value
  kFuStore,                        // X to a dense result
  kFuQuant, kFuQuantY,             // round to dt
  kFuMovYX,                        // Y = X
  kFuAdd, kFuMul, kFuSub, kFuRSub, kFuDiv, kFuRDiv, kFuMax, kFuMin,   // X = X op Y (R: Y op X)
  kFuAddS, kFuMulS, kFuSubS, kFuDivS,                                 // X = X op the row scalar `reg`
  kFuAffine, kFuGelu, kFuGeluGrad, kFuExp, kFuTanh, kFuNeg, kFuSqrt, kFuRsqrt, kFuLog, kFuAbs,   // on X
  kFuGeluGradY,                    // on Y
  kFuRedSum, kFuRedSumSq, kFuRedMax,   // row reduction of X into row scalar `reg`
  kFuSAffine, kFuSRsqrt,           // on row scalar `reg`
  kFuLayerNorm, kFuSoftmax,        // whole-row normalisations of X (s = eps)
  kFuIAdd, kFuISub, kFuIRSub, kFuIMul, kFuIAnd, kFuIOr, kFuIXor, kFuIMax, kFuIMin, kFuUMax, kFuUMin,   // X, Y as 32-bit integers
  kFuINot, kFuINeg,
  kFuCarrySum, kFuCarrySumSq,      // add every X (or its square) to the op's full sum
  kFuEnd
};
constexpr int kFuMaxSteps = 40;
constexpr int kFuScalars = 2;      // row scalars
struct DFuStep {
  uint32_t code, dt;
  float s, t;
  BufRef ptr;
  uint32_t reg, slot;              // row scalar; staging slot of a dense load / row vector (kFuNoSlot: none)
};
constexpr uint32_t kFuNoSlot = 0xFFFFFFFFu;
static_assert(sizeof(DFuStep) == 32, "DFuStep layout");
// A step list that is one of the common row pipelines (ops_rowpipe.cuh), its stages in this order.
enum PipeFlags : uint32_t {
  kRpOn = 1u, kRpRes = 2u, kRpLn = 4u, kRpRms = 8u, kRpMul = 16u, kRpAdd = 32u, kRpGelu = 64u, kRpSoftmax = 128u, kRpCarry = 256u,
  kRpQ = 512u                      // round to the storage type after every stage (else only the result)
};
// Dynamic shared memory of a lane on every device this is built for, and what of it a planned op may stage data in
// (ops_fuse.cuh checks what the interpreter and the step lists take in front).
constexpr uint32_t kLaneSmemBytes = 226u * 1024u, kPlanStageBytes = kLaneSmemBytes - 12u * 1024u;
// How a row pipeline lies over the threads of a lane with `rows` rows: T threads per row, G groups of 4 elements per thread
// (only X lives in registers: up to 8), more threads when rows are few. f32 rows with a residual are staged twice: 8 groups
// of those would be two buffers of 128 KB, so they take 4, and past 8192 columns (512 threads x 16) no row pipeline at all.
struct PipeShape { uint32_t T, G, buf_bytes; };      // buf_bytes: one row of every group, staged
B2_HOST_DEVICE inline PipeShape pipe_shape(uint32_t flags, uint32_t esz, bool vec, uint32_t cols, uint32_t rows, uint32_t nthr) {
  const bool two = (flags & kRpRes) != 0u;
  const uint32_t most = two && esz == 4u ? 16u : 32u;
  PipeShape s;
  s.T = 32u;
  while (s.T < 512u && (cols > s.T * most || rows * s.T * 2u <= nthr)) s.T *= 2u;
  const uint32_t per = (cols + 4u * s.T - 1u) / (4u * s.T);
  s.G = per <= 1u ? 1u : per <= 2u ? 2u : per <= 4u ? 4u : 8u;
  s.buf_bytes = vec ? (two ? 2u : 1u) * s.G * nthr * 4u * esz : 0u;
  return s;
}
struct DPipe {
  uint32_t flags, dt;
  float eps, s, t;
  uint32_t pad;
  BufRef x, y, mul, add, mid, out;
};
// Header of a fused-rows task's descriptor; the steps follow.
struct DFuse {
  uint32_t rows, cols, n_steps;
  uint32_t vec;                    // cols % 4 == 0: 4 consecutive elements per thread and group
  BufRef total;                    // where the full sum goes (kFuCarry*), 0 = none
  uint32_t n_owner_lanes;          // lanes that take part in the full sum
  DPipe pipe;                      // flags != 0: the rows run as this pipeline
  uint32_t n_elems;                // rows x cols, or less where the last "row" of a flat list of elements is short
  uint32_t flat;                   // > 0: a straight chain of so many binary ops on 4-byte elements (ops_flatpipe.cuh)
};
static_assert(sizeof(DFuse) % 8 == 0, "steps follow");
// All-pairs task: the tail is a list of elementwise ops over the n x 3 result, run by the lane on its own rows.
constexpr int kPairTailMax = 24;
// a_src / b_src: 0 = the buffer, 1 = the pair sum itself, 2 + k = what tail op k made
struct DPairTail { uint32_t sub, a_src, b_src, pad; float s, t; BufRef dst, a, b; };
struct DPairs {
  uint32_t n, n_tail;
  float s, t;                      // the affine on the squared distance
  BufRef pos, mass, out;
  DPairTail tail[kPairTailMax];
};

// ---- matmuls ------------------------------------------------------------------------------
// What happens to an accumulated element, in this order.
enum GemmEpi_ : uint32_t {
  kGeQuant0 = 1u,          // round to the product's own 16-bit type (and, with out0, store it)
  kGeGelu = 2u,
  kGeScale0 = 4u,          // times s0
  kGeMaxS = 8u,            // max with s1
  kGeRes = 16u,            // with the residual's element:
  kGeResAdd = 0u << 8, kGeResSub = 1u << 8, kGeResRSub = 2u << 8, kGeResMul = 3u << 8, kGeResGeluGrad = 4u << 8, kGeResMask = 7u << 8,
  kGeCarrySq = 32u,        // add its square to the task's full sum
  kGeScale1 = 64u          // times s1
};
// Epilogues that have a form of their own on the device (ops_gemm.cuh): what a layer leaves after a product going forward (itself, GELU,
// a sum with a residual) and in a training step (GELU's derivative, the update, the loss). Every form is code in each build with
// products; the rest, and what leaves as f32 or in rows that are no whole 16-byte words, takes the general epilogue (4096 x 4096 by
// K = 1024 times an array 62 us, plus one by its form 47; as f32 50, as bf16 by its form 37). kGfF16 is added for f16.
enum GemmForm : uint32_t { kGfAny = 0, kGfPlain, kGfGelu, kGfAdd, kGfGrad, kGfStep, kGfLoss, kGfF16 = 16 };
// One 16-bit type throughout, whole 16-byte words, and a second result only where a form stores it.
inline uint32_t gemm_form_of(uint32_t epi, uint32_t N, bool out0, bool out1, uint32_t dt0, uint32_t dt1, uint32_t qdt, uint32_t rdt) {
  if (!out1 || (dt1 != kBF16 && dt1 != kF16) || N % 8u || ((epi & kGeQuant0) && qdt != dt1) || ((epi & kGeRes) && rdt != dt1)) return kGfAny;
  uint32_t form;
  switch (epi & ~kGeQuant0) {
    case 0u: form = kGfPlain; break;                               // (the store rounds)
    case kGeGelu: form = kGfGelu; break;
    case kGeRes | kGeResAdd: form = kGfAdd; break;
    case kGeRes | kGeResGeluGrad: form = kGfGrad; break;
    case kGeScale0 | kGeRes | kGeResRSub: form = kGfStep; break;
    case kGeRes | kGeResSub | kGeCarrySq | kGeScale1: form = kGfLoss; break;
    default: return kGfAny;
  }
  if (out0 && !(form == kGfGelu && (epi & kGeQuant0) && dt0 == dt1)) return kGfAny;
  return form + (dt1 == kF16 ? kGfF16 : 0u);
}
// unit stride along k; along the rows / columns (MN), fetched as a box of 64-row blocks or block by block
enum GemmOperand : uint32_t { kGmK = 0, kGmMnBlocks = 1, kGmMnSingle = 2 };
struct DGemmProb {
  uint32_t first, tm, tn;          // number of its first tile; tile grid
  uint32_t halves, bn;             // a tile is halves x 128 rows by bn columns
  uint32_t M, N, K;
  uint32_t amn, bmn;               // how an operand lies and is fetched (kGm*)
  uint32_t adt, dt0, dt1;
  int32_t tmap;
  uint32_t epi, qdt, rdt;
  float s0, s1, gg;                // gg: the GELU derivative's free constant
  uint32_t form, pad;              // GemmForm
  BufRef res, out0, out1;
};
constexpr int kGemmMaxProbs = 6;
constexpr uint32_t kGemmRing = 196608, kGemmStagesMax = 8;
struct DGemm {
  uint32_t n_prob, tiles;
  BufRef total;
  uint32_t n_owner_lanes;
  uint32_t stages, stage_bytes;    // of the ring: one holds 64 k of the task's largest tile
  uint32_t pad;
  DGemmProb prob[kGemmMaxProbs];
};

// Products on the CUDA cores. An operand's element (row or column r, k) sits at off + r rs + k ks (elements), or
// through a view where an axis is not affine: at a row's part + a k's part.
enum SgMode : uint32_t { kSgScalar = 0, kSgVecR = 1 };     // element by element; f32, fours of neighbouring rows
struct DSgOperand {
  BufRef ptr;
  uint32_t mode, k_fast;           // element by element: neighbouring threads take neighbouring k (else neighbouring rows)
  uint32_t off, rs, ks;
  uint32_t viewed, row_major, inner;   // view over [rows, k] (row_major) or [k, rows], `inner` = its second extent
  DView v;
};
struct DSgemm {
  uint32_t M, N, K, adt;
  uint32_t shape, epi, qdt, rdt;
  float s0, s1, gg;
  uint32_t n_owner_lanes;
  BufRef res, out0, out1, total;
  uint32_t dt0, dt1;
  DSgOperand a, b;
  // kTopSkinny: A is the RMS norm of the rows at a.ptr: x rsqrt(ns sum x^2 + nt) gamma (0: A as it is)
  BufRef gamma;
  float ns, nt;
  uint32_t move, pad;      // kTopSkinny: out1 is written through this dynamic slice (desc index of its DMove; 0: dense)
};

}  // namespace b2
#endif
