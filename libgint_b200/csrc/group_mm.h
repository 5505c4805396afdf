// group_mm.h -- launcher of k_group_mm (group_mm.cu), the group kernel of the classes without
// generated group code.
#pragma once
#include <cuda_runtime.h>
#include "kernels.h"

namespace gint {

// The classes are instantiated in kMmParts translation units (group_mm.cu compiled with
// GROUP_MM_PART = 0..kMmParts-1) so that they compile in parallel.
constexpr int kMmParts = 11;
constexpr int kMmStaticBytes = 1024;   // shared memory that the kernel declares itself, rounded up

// spherical functions and shared-memory limits on the current device (smax: its opt-in shared memory
// per block; c2s: [4][70] as in upload_constant_tables)
cudaError_t group_mm_preload(int smax, const double *c2s);
// launches class bt.cls, cudaErrorInvalidValue if it has generated group code
cudaError_t group_mm_launch(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st);

#define GROUP_MM_DECL(i)                                                                       \
   cudaError_t group_mm_part##i(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st);      \
   cudaError_t group_mm_preload_part##i(int dyn, const double *c2s);
GROUP_MM_DECL(0) GROUP_MM_DECL(1) GROUP_MM_DECL(2) GROUP_MM_DECL(3) GROUP_MM_DECL(4) GROUP_MM_DECL(5)
GROUP_MM_DECL(6) GROUP_MM_DECL(7) GROUP_MM_DECL(8) GROUP_MM_DECL(9) GROUP_MM_DECL(10)
#undef GROUP_MM_DECL

}  // namespace gint
