// group_mm.h -- launcher of k_group_mm (group_mm.cu), the group kernel of the classes without
// generated group code.
#pragma once
#include <cuda_runtime.h>
#include <vector>
#include "engine_types.h"
#include "kernels.h"

namespace gint {

struct MmDims;
constexpr int kMmTabStride = 74;       // functions of the largest pair, (ff|: e = 3..6
constexpr int kMmStaticBytes = 1024;   // shared memory that the kernel declares itself, rounded up

// the HRR and spherical transform of all 16 shell pairs: coefficients, and per pair and function e
// {first coefficient, first monomial << 8 | monomials}
void group_mm_build(const double *c2s, std::vector<double> &coef, std::vector<int2> &tab);
// tables and shared-memory limits on the current device (smax: its opt-in shared memory per block)
cudaError_t group_mm_preload(int smax, const double *c2s);
cudaError_t group_mm_launch(const DevCtx &ctx, const BatchArgs &bt, const ClassPlan &hp, int smax, cudaStream_t st);

#define GROUP_MM_DECL(i)                                                                                        \
   cudaError_t group_mm_part##i(const DevCtx &ctx, const BatchArgs &bt, const MmDims &dm, int lb, dim3 grid,    \
                                int threads, cudaStream_t st);                                                  \
   cudaError_t group_mm_preload_part##i(int dyn);
GROUP_MM_DECL(0) GROUP_MM_DECL(1) GROUP_MM_DECL(2) GROUP_MM_DECL(3)
#undef GROUP_MM_DECL

}  // namespace gint
