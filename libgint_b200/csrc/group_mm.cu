// group_mm.cu -- instances, tables and launches of k_group_mm (group_mm.cuh).
//
// Compiled kMmParts times (GROUP_MM_PART = 0..3); part i instantiates the bra shells with la = i.
#include <cuda_runtime.h>
#include <algorithm>
#include <vector>
#include "group_mm.cuh"
#include "group_mm.h"

#ifndef GROUP_MM_PART
#define GROUP_MM_PART 0
#endif

namespace gint {
namespace {

template <int LB>
cudaError_t launch_lb(const DevCtx &ctx, const BatchArgs &bt, const MmDims &dm, dim3 grid, int threads, cudaStream_t st) {
   k_group_mm<GROUP_MM_PART, LB><<<grid, threads, (size_t)dm.total * 8, st>>>(ctx, bt, dm);
   return cudaGetLastError();
}

template <int LB>
cudaError_t preload_lb(int dyn) {
   return cudaFuncSetAttribute(k_group_mm<GROUP_MM_PART, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn);
}

}  // namespace

#define MM_CAT2(a, b) a##b
#define MM_CAT(a, b) MM_CAT2(a, b)
cudaError_t MM_CAT(group_mm_part, GROUP_MM_PART)(const DevCtx &ctx, const BatchArgs &bt, const MmDims &dm, int lb,
                                                 dim3 grid, int threads, cudaStream_t st) {
   switch (lb) {
      case 0: return launch_lb<0>(ctx, bt, dm, grid, threads, st);
      case 1: return launch_lb<1>(ctx, bt, dm, grid, threads, st);
      case 2: return launch_lb<2>(ctx, bt, dm, grid, threads, st);
      default: return launch_lb<3>(ctx, bt, dm, grid, threads, st);
   }
}

cudaError_t MM_CAT(group_mm_preload_part, GROUP_MM_PART)(int dyn) {
   cudaError_t e;
   if ((e = preload_lb<0>(dyn)) != cudaSuccess || (e = preload_lb<1>(dyn)) != cudaSuccess ||
       (e = preload_lb<2>(dyn)) != cudaSuccess || (e = preload_lb<3>(dyn)) != cudaSuccess)
      return e;
   return cudaSuccess;
}

#if GROUP_MM_PART == 0
namespace {

int nc(int l) { return (l + 1) * (l + 2) / 2; }
void exps(int l, int i, int e[3]) {
   int a = 0;
   while ((a + 1) * (a + 2) / 2 <= i) a++;
   e[0] = l - a; e[2] = i - a * (a + 1) / 2; e[1] = a - e[2];
}
int index_of(const int e[3]) { const int a = e[1] + e[2]; return a * (a + 1) / 2 + e[2]; }

struct Tables {
   double *coef = nullptr;
   int2 *tab = nullptr;
   uint16_t *tmap = nullptr;
};
Tables g_tables[kMaxDevices];

// the places of the targets of class c in T, back to back over the classes
int tmap_first(int cls) {
   static const std::vector<int> first = [] {
      std::vector<int> f(257, 0);
      ClassPlan p;
      for (int c = 0; c < 256; c++) {
         build_class_plan(c >> 6, (c >> 4) & 3, (c >> 2) & 3, c & 3, p);
         f[c + 1] = f[c] + p.S;
      }
      return f;
   }();
   return first[cls];
}

int sum_cart(int l0, int l1) { int n = 0; for (int l = l0; l <= l1; l++) n += nc(l); return n; }

}  // namespace

// B of a bra (a b|: the HRR gives (a b| = sum over beta <= b of binomial(b, beta) (A - B)^(b - beta)
// (a + beta|, componentwise (the closed form of reference src/compute_HRR.cpp:7-99), and the
// spherical rows are sums of cartesian pairs. The element of (ma mb) and e = a + beta is thus a
// homogeneous polynomial of degree b - beta in A - B, stored as its coefficients over all monomials
// of that degree. The ket's K is the same with C - D.
void group_mm_build(const double *c2s, std::vector<double> &coef, std::vector<int2> &tab) {
   static const int first_mono[4] = {0, 1, 4, 10}, binom[4][4] = {{1, 0, 0, 0}, {1, 1, 0, 0}, {1, 2, 1, 0}, {1, 3, 3, 1}};
   coef.clear();
   tab.assign(16 * kMmTabStride, make_int2(0, 0));
   for (int la = 0; la <= 3; la++)
      for (int lb = 0; lb <= 3; lb++) {
         int x = 0;
         for (int le = la; le <= la + lb; le++)
            for (int e = 0; e < nc(le); e++, x++) {
               const int deg = la + lb - le, nm = nc(deg);
               int ex[3];
               exps(le, e, ex);
               const int ng = (2 * la + 1) * (2 * lb + 1);
               const size_t first = coef.size();   // [monomial][ma mb]
               tab[(la * 4 + lb) * kMmTabStride + x] = make_int2((int)first, (first_mono[deg] << 8) | nm);
               coef.resize(first + (size_t)nm * ng);
               for (int ma = 0; ma < 2 * la + 1; ma++)
                  for (int mb = 0; mb < 2 * lb + 1; mb++) {
                     double m[10] = {0};
                     for (int ca = 0; ca < nc(la); ca++)
                        for (int cb = 0; cb < nc(lb); cb++) {
                           int ea[3], eb[3], left[3];
                           exps(la, ca, ea);
                           exps(lb, cb, eb);
                           double f = c2s[la * 70 + ma * nc(la) + ca] * c2s[lb * 70 + mb * nc(lb) + cb];
                           bool ok = f != 0.0;
                           for (int d = 0; d < 3 && ok; d++) {
                              const int beta = ex[d] - ea[d];
                              ok = beta >= 0 && beta <= eb[d];
                              if (ok) { f *= binom[eb[d]][beta]; left[d] = eb[d] - beta; }
                           }
                           if (ok) m[index_of(left)] += f;
                        }
                     for (int k = 0; k < nm; k++) coef[first + (size_t)k * ng + ma * (2 * lb + 1) + mb] = m[k];
                  }
            }
      }
}

cudaError_t group_mm_preload(int smax, const double *c2s) {
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
   cudaError_t (*parts[])(int) = {group_mm_preload_part0, group_mm_preload_part1, group_mm_preload_part2, group_mm_preload_part3};
   for (auto f : parts)
      if ((e = f(smax - kMmStaticBytes)) != cudaSuccess) return e;
   if (g_tables[dev].coef) return cudaSuccess;
   std::vector<double> coef;
   std::vector<int2> tab;
   group_mm_build(c2s, coef, tab);
   std::vector<uint16_t> tmap((size_t)tmap_first(256));
   ClassPlan p;
   for (int c = 0; c < 256; c++) {
      build_class_plan(c >> 6, (c >> 4) & 3, (c >> 2) & 3, c & 3, p);
      const int FP = (sum_cart(p.lc, p.lc + p.ld) + 3) & ~3;
      uint16_t *t = tmap.data() + tmap_first(c);
      int f0 = 0, s = 0;   // a panel [nE][ncart(f)] per ket shell f
      for (int f = p.lc; f <= p.lc + p.ld; f0 += nc(f), f++)
         for (int x = 0; x < p.nE; x++)
            for (int k = 0; k < nc(f); k++) t[s++] = (uint16_t)(x * FP + f0 + k);
   }
   Tables T;
   if ((e = cudaMalloc(&T.coef, coef.size() * 8)) == cudaSuccess && (e = cudaMalloc(&T.tab, tab.size() * sizeof(int2))) == cudaSuccess &&
       (e = cudaMalloc(&T.tmap, tmap.size() * 2)) == cudaSuccess &&
       (e = cudaMemcpy(T.coef, coef.data(), coef.size() * 8, cudaMemcpyHostToDevice)) == cudaSuccess &&
       (e = cudaMemcpy(T.tab, tab.data(), tab.size() * sizeof(int2), cudaMemcpyHostToDevice)) == cudaSuccess)
      e = cudaMemcpy(T.tmap, tmap.data(), tmap.size() * 2, cudaMemcpyHostToDevice);
   if (e != cudaSuccess) {
      cudaFree(T.coef); cudaFree(T.tab); cudaFree(T.tmap);
      return e;
   }
   g_tables[dev] = T;
   return cudaSuccess;
}

// the least stride >= n that is 4 modulo 16 doubles: eight rows by four columns of doubles then
// fall on different banks
static int stride4(int n) { return n + ((4 - n) & 15); }

cudaError_t group_mm_launch(const DevCtx &ctx, const BatchArgs &bt, const ClassPlan &hp, int smax, cudaStream_t st) {
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices || !g_tables[dev].coef) return cudaErrorInvalidDevice;
   const Tables &T = g_tables[dev];
   const int NA = 2 * hp.la + 1, NB = 2 * hp.lb + 1;
   const int AC = NA <= 3 || NB == 1 ? NA : (NA == 5 ? 3 : 4), NCH = (NA + AC - 1) / AC;   // MmShape
   MmDims dm;
   dm.S = hp.S; dm.nE = hp.nE;
   dm.nF = sum_cart(hp.lc, hp.lc + hp.ld);
   dm.nC = 2 * hp.lc + 1; dm.nD = 2 * hp.ld + 1;
   const int nCD = dm.nC * dm.nD;
   dm.FP = (dm.nF + 3) & ~3;
   dm.CT = (nCD + 7) / 8;
   dm.CS = stride4(dm.CT * 8);
   dm.TS = stride4(dm.nE * dm.FP);
   dm.IS = (NA * NB * nCD) | 1;
   dm.oB = 0;
   dm.oK = dm.oB + dm.nE * NCH * ((AC * NB + 1) & ~1);
   dm.oW = dm.oK + dm.FP * dm.CS;
   dm.oT = dm.oW + kMmPrims * kMmCoefStride;
   // eight rows a tile (the height of a product), fewer where two blocks would not fit an SM
   const int PS = ctx.nspin * (NA + NB) * (dm.nC + dm.nD);
   for (dm.RT = 8; dm.RT > 1 && (dm.oT + dm.RT * (dm.TS + dm.IS + PS)) * 8 > 100 * 1024; dm.RT /= 2) {}
   dm.oI = dm.oT + dm.RT * dm.TS;
   dm.oP = dm.oI + dm.RT * dm.IS;
   dm.total = dm.oP + dm.RT * PS;
   if (dm.total * 8 > smax - kMmStaticBytes) return cudaErrorInvalidConfiguration;
   dm.tmap = T.tmap + tmap_first(bt.cls);
   dm.coef = T.coef;
   dm.btab = T.tab + (hp.la * 4 + hp.lb) * kMmTabStride;
   dm.ktab = T.tab + (hp.lc * 4 + hp.ld) * kMmTabStride;
   // A warp per tile of kets and part of the bras, and per 32 targets; but where groups fill the GPU,
   // 128 threads for all except the largest shapes: more blocks then fit an SM, and the registers of
   // the wide shapes allow two blocks of 128 threads but one of 160 (on the 1/4096 sample of the
   // 64-molecule l <= 3 workload, kernels one after another: 49.0 -> 47.0 ms; with few groups, 2
   // molecules and 27 images, the wider blocks are faster: 13.9 against 18.4 ms).
   const bool many = bt.ngroup >= 148u * 8;
   const int threads = many && (dm.S < 400 || AC * NB > 15)
                           ? 128 : std::max(64, std::min(kMmThreads, 32 * std::max(dm.CT * NCH, (dm.S + 31) / 32)));
   // every block clears the paddings of its products once, so it takes several groups where there are
   // many; where there are too few to fill the GPU, the tiles of a group are dealt out over blocks
   const unsigned y = bt.ngroup < 148 * 4 ? 8 : (bt.ngroup < 148 * 16 ? 2 : 1);
   const dim3 grid(std::min(bt.ngroup, 148u * 32), y);
   switch (hp.la) {
      case 0: return group_mm_part0(ctx, bt, dm, hp.lb, grid, threads, st);
      case 1: return group_mm_part1(ctx, bt, dm, hp.lb, grid, threads, st);
      case 2: return group_mm_part2(ctx, bt, dm, hp.lb, grid, threads, st);
      default: return group_mm_part3(ctx, bt, dm, hp.lb, grid, threads, st);
   }
}
#endif

}  // namespace gint
