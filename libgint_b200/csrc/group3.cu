// group3.cu -- k_group3<la,lb,lc,ld>: contraction + HRR + image-pair sum + spherical transform +
// K update, one lane (or four) per contraction row, for the classes with generated HRR code (grp_gen.cuh).
//
// A group is one set quartet of one class: all its image pairs (shell quartets) and its
// nla*nlb*nlc*nld contraction rows. One lane takes one row: it contracts the image-summed targets
// of each shell over its primitives with the row's coefficients, applies that shell's HRR (its own
// AB and CD), sums the shells, transforms the sum to spherical harmonics and adds the four exchange
// updates to K with atomics (reference src/compute_ECO.cpp:12-214, src/compute_HRR.cpp:102-225,
// src/compute_SPH.cpp:58-237, src/compute_KS.cpp:8-117). All indices are compile-time
// constants and the workspace lives in registers.
//
// Compiled kGroup3Parts times (GROUP3_PART = 0..3); part i instantiates the generated classes
// whose position in kGrpGenClasses is i modulo kGroup3Parts.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "engine_types.h"
#include "grp_gen.cuh"
#include "group3.h"
#include "kernels.h"
#include "prim_common.cuh"

#ifndef GROUP3_PART
#define GROUP3_PART 0
#endif

namespace gint {
namespace {

// symmetry factors by bucket (reference src/libGint.cpp:262-267)
__device__ __forceinline__ double symm_factor(int i) {
   return i == 0 ? 2.0 : (i == 1 ? 1.0 : (i == 2 ? 0.5 : (i == 3 ? 0.25 : 0.0)));
}

// One spin's K update of one row from its spherical block I (reference src/compute_KS.cpp:26-115):
// K_bd -= f I P_ac and its three partners, each summed over the block in registers first. A row of
// (pp|ps) then reads 24 elements of P and adds 24 to K, where one read and one atomic per integral and
// partner were 108 of each (classes of L <= 3 of the 1/4096 sample of the 64-molecule l <= 3 workload,
// with the displacements read instead of derived: 14.1 to 12.9 ms).
template <int NA, int NB, int NC, int ND, class R>
static __device__ __forceinline__ void k_update(const R *I, const double *__restrict__ P, double *K, const QrttRec &k,
                                                double f) {
   // the element (x, y) of pair u (ac, ad, bc, bd) is at off[u] + x sx[u] + y sy[u]
   int sx[4], sy[4];
#pragma unroll
   for (int u = 0; u < 4; u++) {
      const bool T = (k.T >> u) & 1;
      sx[u] = T ? (int)k.ld[u] : 1;
      sy[u] = T ? 1 : (int)k.ld[u];
   }
   // all of P first: one round of independent loads
   double Pac[NA][NC], Pad[NA][ND], Pbc[NB][NC], Pbd[NB][ND];
#pragma unroll
   for (int a = 0; a < NA; a++) {
#pragma unroll
      for (int c = 0; c < NC; c++) Pac[a][c] = __ldg(P + ((size_t)k.off[0] + a * sx[0] + c * sy[0]));
#pragma unroll
      for (int d = 0; d < ND; d++) Pad[a][d] = __ldg(P + ((size_t)k.off[1] + a * sx[1] + d * sy[1]));
   }
#pragma unroll
   for (int b = 0; b < NB; b++) {
#pragma unroll
      for (int c = 0; c < NC; c++) Pbc[b][c] = __ldg(P + ((size_t)k.off[2] + b * sx[2] + c * sy[2]));
#pragma unroll
      for (int d = 0; d < ND; d++) Pbd[b][d] = __ldg(P + ((size_t)k.off[3] + b * sx[3] + d * sy[3]));
   }
#define I4(a, b, c, d) ((double)I[(((a) * NB + (b)) * NC + (c)) * ND + (d)])
#pragma unroll
   for (int b = 0; b < NB; b++) {
#pragma unroll
      for (int d = 0; d < ND; d++) {
         double v = 0.0;
#pragma unroll
         for (int a = 0; a < NA; a++)
#pragma unroll
            for (int c = 0; c < NC; c++) v += I4(a, b, c, d) * Pac[a][c];
         atomicAdd(K + ((size_t)k.off[3] + b * sx[3] + d * sy[3]), f * v);
      }
#pragma unroll
      for (int c = 0; c < NC; c++) {
         double v = 0.0;
#pragma unroll
         for (int a = 0; a < NA; a++)
#pragma unroll
            for (int d = 0; d < ND; d++) v += I4(a, b, c, d) * Pad[a][d];
         atomicAdd(K + ((size_t)k.off[2] + b * sx[2] + c * sy[2]), f * v);
      }
   }
#pragma unroll
   for (int a = 0; a < NA; a++) {
#pragma unroll
      for (int d = 0; d < ND; d++) {
         double v = 0.0;
#pragma unroll
         for (int b = 0; b < NB; b++)
#pragma unroll
            for (int c = 0; c < NC; c++) v += I4(a, b, c, d) * Pbc[b][c];
         atomicAdd(K + ((size_t)k.off[1] + a * sx[1] + d * sy[1]), f * v);
      }
#pragma unroll
      for (int c = 0; c < NC; c++) {
         double v = 0.0;
#pragma unroll
         for (int b = 0; b < NB; b++)
#pragma unroll
            for (int d = 0; d < ND; d++) v += I4(a, b, c, d) * Pbd[b][d];
         atomicAdd(K + ((size_t)k.off[0] + a * sx[0] + c * sy[0]), f * v);
      }
   }
#undef I4
}

// resident 128-thread blocks per SM the register budget is sized for: the kernel waits on
// chains of dependent loads, so small classes trade registers for more warps in flight
template <int LA, int LB, int LC, int LD>
struct Group3Shape {
   static constexpr int L = LA + LB + LC + LD;
   static constexpr int MINB = L <= 1 ? 8 : (L == 2 ? 6 : 4);
};

// R = double: the FP64 path; R = float: the FP32 path (contraction, HRR and spherical transform in
// FP32 from the FP32 targets of k_prim3; the K update in FP64).
// TPR lanes share one contraction row: they divide its targets, and all go on with all of them.
template <int LA, int LB, int LC, int LD, class R, int TPR>
__global__ void __launch_bounds__(128, Group3Shape<LA, LB, LC, LD>::MINB / (TPR == 1 ? 1 : 2)) k_group3(DevCtx ctx, BatchArgs bt) {
   using G = GrpGen<LA, LB, LC, LD>;
   constexpr int S = G::S, Nc = G::Nc, Ns = G::Ns;
   const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
   constexpr int RPW = 32 / TPR;   // rows a warp
   const uint32_t nblk = (bt.nqrtt + RPW - 1) / RPW;
   const int sub = lane % TPR;
   const unsigned team = TPR == 1 ? 1u << lane : ((1u << TPR) - 1u) << (lane - sub);
   // a warp takes RPW consecutive rows, so the lanes of one set quartet's rows read the same
   // primitive codes and image-summed targets (broadcast loads)
   for (uint32_t blk = blockIdx.x * wpb + (threadIdx.x >> 5); blk < nblk; blk += gridDim.x * wpb) {
      const uint32_t q0 = blk * RPW, q = q0 + lane / TPR;
      uint32_t gi = row_group_warp(bt, q0 & ~31u, lane);
      if (TPR > 1) gi = __shfl_sync(0xffffffffu, gi, (int)(q0 & 31u) + lane / TPR);
      if (q >= bt.nqrtt || (bt.gflags && !__ldg(bt.gflags + gi))) continue;   // screened (incremental)
      const GroupRec Gr = bt.groups[gi];
      const int nl1 = Gr.nl[1], nl2 = Gr.nl[2], nl3 = Gr.nl[3];
      const int r = (int)(q - Gr.qrtt_off);
      const int ia = r / (nl1 * nl2 * nl3), ib = (r / (nl2 * nl3)) % nl1, ic = (r / nl3) % nl2, id = r % nl3;
      R cart[Nc];
#pragma unroll
      for (int t = 0; t < Nc; t++) cart[t] = R(0);
      for (uint32_t s = 0; s < Gr.nshell; s++) {
         const ShellRec sh = bt.shells[Gr.shell_off + s];
         const BasisEnt &ea = ctx.ents[sh.ent[0]], &eb = ctx.ents[sh.ent[1]];
         const BasisEnt &ec = ctx.ents[sh.ent[2]], &ed = ctx.ents[sh.ent[3]];
         const double *Ka = ctx.pool + ea.k_off + ia * ea.np;
         const double *Kb = ctx.pool + eb.k_off + ib * eb.np;
         const double *Kc = ctx.pool + ec.k_off + ic * ec.np;
         const double *Kd = ctx.pool + ed.k_off + id * ed.np;
         R T[S];
#pragma unroll
         for (int j = 0; j < S; j++) T[j] = R(0);
         // contraction over the primitives (reference src/compute_ECO.cpp:131-212)
         const R *ac = reinterpret_cast<const R *>(bt.AC) + (size_t)sh.prm_off * S;
         auto coef = [&](uint32_t ip) {
            const uint32_t code = __ldg(bt.prm + sh.prm_off + ip);
            return (R)__ldg(Ka + (code >> 24)) * (R)__ldg(Kb + ((code >> 16) & 255)) * (R)__ldg(Kc + ((code >> 8) & 255)) *
                   (R)__ldg(Kd + (code & 255));
         };
         if constexpr (TPR == 1) {
            // four per iteration so that the next ones' loads overlap this one's FMAs
#pragma unroll 4
            for (uint32_t ip = 0; ip < sh.nprm; ip++) {
               const R kp = coef(ip);
               const R *row = ac + (size_t)ip * S;
#pragma unroll
               for (int j = 0; j < S; j++) T[j] += kp * __ldg(row + j);
            }
         } else {
            // lane `sub` sums targets sub, sub + TPR, ... over the primitives in their order, and makes the
            // coefficient of every TPR-th primitive; the loads of TPR * UP primitives are under way at a time
            constexpr int SQ = (S + TPR - 1) / TPR, UP = SQ <= 2 ? 4 : (SQ <= 4 ? 2 : 1);
            R t[SQ];
#pragma unroll
            for (int i = 0; i < SQ; i++) t[i] = R(0);
            for (uint32_t p0 = 0; p0 < sh.nprm; p0 += TPR * UP) {
               R mine[UP], a[UP][TPR][SQ];
#pragma unroll
               for (int u = 0; u < UP; u++) {
                  mine[u] = p0 + u * TPR + sub < sh.nprm ? coef(p0 + u * TPR + sub) : R(0);
#pragma unroll
                  for (int k = 0; k < TPR; k++)
#pragma unroll
                     for (int i = 0; i < SQ; i++) {
                        const uint32_t ip = p0 + u * TPR + k;
                        a[u][k][i] = ip < sh.nprm && i * TPR + sub < S ? __ldg(ac + (size_t)ip * S + i * TPR + sub) : R(0);
                     }
               }
#pragma unroll
               for (int u = 0; u < UP; u++)
#pragma unroll
                  for (int k = 0; k < TPR; k++) {
                     const R kp = __shfl_sync(team, mine[u], lane - sub + k);
#pragma unroll
                     for (int i = 0; i < SQ; i++) t[i] += kp * a[u][k][i];
                  }
            }
#pragma unroll
            for (int j = 0; j < S; j++) T[j] = __shfl_sync(team, t[j / TPR], lane - sub + j % TPR);
         }
         double v[6];
         read_shell_vectors(ctx, bt, Gr.shell_off + s, sh, v);
         const R AB[3] = {(R)v[0], (R)v[1], (R)v[2]}, CD[3] = {(R)v[3], (R)v[4], (R)v[5]};
         G::hrr(T, AB, CD, cart);
      }
      if (TPR > 1 && sub) continue;
      R sph[Ns];
      G::sph(cart, sph);
      const QrttRec k = bt.qrtts[q];
      const double fac = symm_factor(k.idx_fac) * ctx.hf_fac;
      if (!row_in_range(k, 2 * LA + 1, 2 * LB + 1, 2 * LC + 1, 2 * LD + 1, ctx.FP_size)) {
         atomicOr(ctx.err, 1);
         continue;
      }
      for (int sp = 0; sp < ctx.nspin; sp++)
         k_update<2 * LA + 1, 2 * LB + 1, 2 * LC + 1, 2 * LD + 1>(sph, ctx.P[sp], ctx.K[sp], k, -fac);
   }
}

template <int LA, int LB, int LC, int LD, int TPR>
cudaError_t launch_lanes(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
   const int threads = 128;
   // 32 / TPR rows per warp: rows cost from one primitive to thousands, so the block scheduler, which
   // starts a new block wherever one finishes, balances them better than a grid-stride loop
   const long blocks = std::max(1L, std::min(((long)bt.nqrtt * TPR + threads - 1) / threads, 1L << 30));
   if (bt.fp32) {
      if constexpr (class_has_fp32(LA, LB, LC, LD) && TPR == 1) {
         k_group3<LA, LB, LC, LD, float, 1><<<(unsigned)blocks, threads, 0, st>>>(ctx, bt);
         return cudaGetLastError();
      } else {
         return cudaErrorInvalidValue;   // no FP32 segments for these classes, and none with more lanes
      }
   }
   k_group3<LA, LB, LC, LD, double, TPR><<<(unsigned)blocks, threads, 0, st>>>(ctx, bt);
   return cudaGetLastError();
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_one(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st) {
   // Too few rows to fill half of the warps that the registers leave room for: four lanes a row. (The
   // rows of one set quartet read the same targets, so more lanes a row cost reads where there are
   // rows enough: the line lies where the GPU has nothing else to run.) The classes of L <= 3, kernels one
   // after another: 4 molecules l <= 2 2.70 -> 0.69 ms, 24 clusters 6.85 -> 2.40 ms, 32 molecules
   // l <= 2 2.83 -> 1.04 ms; the 1/4096 sample of 64 molecules, with 150k rows and more a class, unchanged.
   // (Lanes that divided the primitives took 1.03, 2.90 and 1.36 ms, and changed the order of their sum.)
   // FP32 rows keep one lane: there is no FP32 instance of four.
   if (!bt.fp32 && bt.nqrtt < 148u * 64 * Group3Shape<LA, LB, LC, LD>::MINB) return launch_lanes<LA, LB, LC, LD, 4>(ctx, bt, st);
   return launch_lanes<LA, LB, LC, LD, 1>(ctx, bt, st);
}

template <int I>
struct PartTable {
   static bool launch(int cls, const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st, cudaError_t *err) {
      if constexpr (I >= kGrpGenCount) {
         return false;
      } else {
         constexpr int c = kGrpGenClasses[I];
         if (cls == c) {
            *err = launch_one<(c >> 6) & 3, (c >> 4) & 3, (c >> 2) & 3, c & 3>(ctx, bt, st);
            return true;
         }
         return PartTable<I + kGroup3Parts>::launch(cls, ctx, bt, st, err);
      }
   }
};

// loads (and so registers with the runtime) every kernel of this part
template <int I>
struct PartPreload {
   static cudaError_t run() {
      if constexpr (I >= kGrpGenCount) {
         return cudaSuccess;
      } else {
         constexpr int c = kGrpGenClasses[I];
         constexpr int la = (c >> 6) & 3, lb = (c >> 4) & 3, lc = (c >> 2) & 3, ld = c & 3;
         cudaFuncAttributes a;
         cudaError_t e;
         if ((e = cudaFuncGetAttributes(&a, k_group3<la, lb, lc, ld, double, 1>)) != cudaSuccess) return e;
         if ((e = cudaFuncGetAttributes(&a, k_group3<la, lb, lc, ld, double, 4>)) != cudaSuccess) return e;
         if constexpr (class_has_fp32(la, lb, lc, ld)) {
            if ((e = cudaFuncGetAttributes(&a, k_group3<la, lb, lc, ld, float, 1>)) != cudaSuccess) return e;
         }
         return PartPreload<I + kGroup3Parts>::run();
      }
   }
};

}  // namespace

#define GROUP3_CAT2(a, b) a##b
#define GROUP3_CAT(a, b) GROUP3_CAT2(a, b)
bool GROUP3_CAT(group3_launch_part, GROUP3_PART)(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st,
                                                 cudaError_t *err) {
   if (bt.nqrtt == 0) { *err = cudaSuccess; return true; }
   return PartTable<GROUP3_PART>::launch(bt.cls, ctx, bt, st, err);
}

cudaError_t GROUP3_CAT(group3_preload_part, GROUP3_PART)() { return PartPreload<GROUP3_PART>::run(); }

#if GROUP3_PART == 0
cudaError_t group3_preload() {
   cudaError_t (*parts[])() = {group3_preload_part0, group3_preload_part1, group3_preload_part2,
                               group3_preload_part3};
   for (auto f : parts) {
      cudaError_t e = f();
      if (e != cudaSuccess) return e;
   }
   return cudaSuccess;
}

bool group3_launch(const DevCtx &ctx, const BatchArgs &bt, cudaStream_t st, cudaError_t *err) {
   static_assert(kGroup3Parts == 4, "one call per part below");
   return group3_launch_part0(ctx, bt, st, err) || group3_launch_part1(ctx, bt, st, err) ||
          group3_launch_part2(ctx, bt, st, err) || group3_launch_part3(ctx, bt, st, err);
}
#endif

}  // namespace gint
