// Kernel tables of the generation kernels.
//
// Each (entry kind, emission source, normalisation block) triple is
// instantiated in its own translation unit (glp_gen_*.cu) so the
// instantiations compile in parallel; the host code picks a kernel by its
// speculation width: P lanes per sample (P/2 evaluations a round); for one chunk
// also the teams of two and four warps.
#pragma once

#include "glp_kernels.cuh"

namespace glp {

using SingleFn = void (*)(const GenParams);
using MultiFn = void (*)(const MultiParams);

SingleFn single_kernel_f32(uint32_t P);
SingleFn single_kernel_vq(uint32_t P);
MultiFn multi_kernel_f32(uint32_t P);
MultiFn multi_kernel_vq(uint32_t P);
// the same with normalisation every 4 sites
SingleFn single_kernel_f32_sub4(uint32_t P);
SingleFn single_kernel_vq_sub4(uint32_t P);
MultiFn multi_kernel_f32_sub4(uint32_t P);
MultiFn multi_kernel_vq_sub4(uint32_t P);

}  // namespace glp

// Body of one table: KERNEL<P, EMIT, SUB> for P = 2, 4, 8, 16, 32 (narrower
// requests get two lanes: one evaluation a round, the sequential chain) and MORE.
#define GLP_GEN_TABLE(NAME, FNTYPE, KERNEL, EMIT, SUB, MORE) \
  FNTYPE NAME(uint32_t P) {                                  \
    switch (P) {                                             \
      case 0:                                                \
      case 1:                                                \
      case 2: return KERNEL<2, EMIT, SUB>;                   \
      case 4: return KERNEL<4, EMIT, SUB>;                   \
      case 8: return KERNEL<8, EMIT, SUB>;                   \
      case 16: return KERNEL<16, EMIT, SUB>;                 \
        MORE(KERNEL, EMIT, SUB)                              \
      default: return KERNEL<32, EMIT, SUB>;                 \
    }                                                        \
  }
// Teams wider than a block of the build's warps holds (kWidest) are not there.
#define GLP_GEN_TEAMS(KERNEL, EMIT, SUB)                                  \
  case 64: return KERNEL<(kWidest >= 64 ? 64 : 32), EMIT, SUB>;           \
  case 128: return KERNEL<(kWidest >= 128 ? 128 : 32), EMIT, SUB>;
#define GLP_GEN_NO_TEAMS(KERNEL, EMIT, SUB)
