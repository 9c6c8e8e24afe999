// The builds of the megakernel the library carries. Each is the same interpreter
// (vm_kernel.cu) compiled with only some tile-op families present; a program runs
// on the first build in this list that has every family its tasks use, so it does
// not pay (in registers, instruction-cache footprint and compiler decisions) for
// tile ops it never executes. The reference builds its megakernel with a
// compile-time op mask for attribution (VMO_STUB_MASK,
// pjrt_plugin/kernels/vm_main.cl:19-27); here the mask selects what is shipped.
//
// B2_VARIANT_LIST(X) expands X(name, family mask) in order of preference
// (smallest first; `all` holds every family a wire program can name; the ones after
// it hold the re-planner's own ops and run on plan_kernel.cu). The build script
// reads the same list to compile one object per entry.
//
// The builds for decode steps, f32 blocks and 16-bit blocks have the attention with only the products such a program runs: in the
// one build with all of them a batch 32 decode step takes 158 us (148 in its own), an f32 block of width 512 320 us (291).
// The decode build comes before plan_gemm: lone skinny products run on it, where their code keeps more of its values in registers (spilled
// bytes 56 for 244; three of 32 x 1024 by 1024 16.2 us for 17.9, 1 x 4096 by 4096 22.0 for 25.0).
#ifndef B2VM_VARIANTS_H_
#define B2VM_VARIANTS_H_

#include "format.h"

#define B2_FAMS_STREAM (b2::kFamEw | b2::kFamMove | b2::kFamRed | b2::kFamRows | b2::kFamRegion)
#define B2_VARIANT_LIST(X)                               \
  X(stream, B2_FAMS_STREAM)                              \
  X(shortrun, B2_FAMS_STREAM | b2::kFamShort)            \
  X(matmul, B2_FAMS_STREAM | b2::kFamMma)                \
  X(attn, B2_FAMS_STREAM | b2::kFamMma | b2::kFamFlash)  \
  X(all, b2::kFamWire)                                   \
  X(plan_rows, b2::kFamFuse)                             \
  X(plan_pairs, b2::kFamFuse | b2::kFamPairs)            \
  X(plan_decode, b2::kFamFuse | b2::kFamSkinny | b2::kFamFlash | b2::kFamMove) \
  X(plan_gemm, b2::kFamFuse | b2::kFamGemm | b2::kFamSkinny) \
  X(plan_sgemm, b2::kFamFuse | b2::kFamSgemm)            \
  X(plan_f32, b2::kFamFuse | b2::kFamSgemm | b2::kFamFlash | b2::kFamMove) \
  X(plan_block, b2::kFamFuse | b2::kFamGemm | b2::kFamFlash | b2::kFamMove) \
  X(plan_attn, b2::kFamFuse | b2::kFamGemm | b2::kFamSgemm | b2::kFamSkinny | b2::kFamFlash | b2::kFamMove)

#endif
