// group_mm.cu -- instances and launches of k_group_mm (group_mm.cuh).
//
// Compiled kMmParts times (GROUP_MM_PART = 0..kMmParts-1); part i instantiates the classes without
// generated group code whose number la*64 + lb*16 + lc*4 + ld is i modulo kMmParts.
#include <cuda_runtime.h>
#include <algorithm>
#include "group_mm.cuh"
#include "group_mm.h"
#include "grp_gen.cuh"

#ifndef GROUP_MM_PART
#define GROUP_MM_PART 0
#endif

namespace gint {
namespace {

template <int CLS>
cudaError_t launch_one(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
   using Sh = MmShape<CLS>;
   static_assert(Sh::doubles(2) * 8 + kMmStaticBytes <= 227 * 1024, "two spins fit a block's shared memory");
   // 128 threads: more blocks fit an SM than of 256, except where a row is worked on by the whole block, or
   // groups are so few that their chains of stages are the whole time (replays with 128 and with 256
   // threads for all: 64 molecules l <= 3, 1/4096, 58.1 and 67.3 ms; 24 clusters, mostly 10 to 200 groups
   // a class, 4.24 and 5.05 ms; 2 molecules and 27 images, up to 32 groups a class, 1.75 and 1.61 ms)
   const int threads = Sh::kWide || bt.ngroup < 64 ? kMmThreads : 128;
   // where there are too few groups to fill the GPU, the tiles of a group are dealt out over blocks
   // (2 molecules and 27 images, all of a group's tiles to one block: 2.32 instead of 1.61 ms)
   const unsigned y = bt.ngroup < 148 * 4 ? 8 : (bt.ngroup < 148 * 16 ? 2 : 1);
   k_group_mm<CLS><<<dim3(std::min(bt.ngroup, 148u * 32), y), threads, (size_t)Sh::doubles(ctx.nspin) * 8, st>>>(ctx, bt);
   return cudaGetLastError();
}

// the classes of this part from CLS on
template <int CLS>
struct Part {
   static cudaError_t launch(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
      if constexpr (CLS >= 256) {
         return cudaErrorInvalidValue;
      } else {
         if constexpr (!GrpGen<(CLS >> 6) & 3, (CLS >> 4) & 3, (CLS >> 2) & 3, CLS & 3>::kHas)
            if (bt.cls == CLS) return launch_one<CLS>(ctx, bt, st);
         return Part<CLS + kMmParts>::launch(ctx, bt, st);
      }
   }
   static cudaError_t preload(int dyn) {
      if constexpr (CLS >= 256) {
         return cudaSuccess;
      } else {
         if constexpr (!GrpGen<(CLS >> 6) & 3, (CLS >> 4) & 3, (CLS >> 2) & 3, CLS & 3>::kHas) {
            const cudaError_t e = cudaFuncSetAttribute(k_group_mm<CLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
            if (e != cudaSuccess) return e;
         }
         return Part<CLS + kMmParts>::preload(dyn);
      }
   }
};

}  // namespace

#define MM_CAT2(a, b) a##b
#define MM_CAT(a, b) MM_CAT2(a, b)
cudaError_t MM_CAT(group_mm_part, GROUP_MM_PART)(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
   return Part<GROUP_MM_PART>::launch(ctx, bt, st);
}

cudaError_t MM_CAT(group_mm_preload_part, GROUP_MM_PART)(int dyn, const double *c2s) {
   const cudaError_t e = cudaMemcpyToSymbol(c_mm_c2s, c2s, sizeof(c_mm_c2s));
   return e != cudaSuccess ? e : Part<GROUP_MM_PART>::preload(dyn);
}

#if GROUP_MM_PART == 0
cudaError_t group_mm_preload(int smax, const double *c2s) {
   cudaError_t (*parts[kMmParts])(int, const double *) = {
       group_mm_preload_part0, group_mm_preload_part1, group_mm_preload_part2, group_mm_preload_part3,
       group_mm_preload_part4, group_mm_preload_part5, group_mm_preload_part6, group_mm_preload_part7,
       group_mm_preload_part8, group_mm_preload_part9, group_mm_preload_part10};
   for (auto f : parts) {
      const cudaError_t e = f(smax - kMmStaticBytes, c2s);
      if (e != cudaSuccess) return e;
   }
   return cudaSuccess;
}

cudaError_t group_mm_launch(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
   cudaError_t (*parts[kMmParts])(const DevCtx &, const BatchArgs &, cudaStream_t) = {
       group_mm_part0, group_mm_part1, group_mm_part2, group_mm_part3, group_mm_part4, group_mm_part5,
       group_mm_part6, group_mm_part7, group_mm_part8, group_mm_part9, group_mm_part10};
   return parts[bt.cls % kMmParts](ctx, bt, st);
}
#endif

}  // namespace gint
