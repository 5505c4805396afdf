// group_mm.cuh -- k_group_mm<class>: contraction, HRR, image-pair sum, spherical transform and K
// update of the classes without generated group code, one block per set quartet.
//
// The contraction is a dense product (rows x primitives times primitives x targets) on the FP64
// tensor cores, whose m8n8k4 product rounds as a chain of fused multiply-adds in the order of k: a
// target is summed over its primitives in their order, as one lane of the other group kernels does.
// The HRR then runs in registers and element for element by the recursion of those kernels
// (reference src/compute_HRR.cpp:7-99): an element of (a b| is a difference of terms |A - B|^b times
// larger, so that another order of its sums shows in K (4e-8 of K's root mean square on the 64-molecule
// l <= 3 workload), and all group kernels keep to one.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include <utility>
#include "engine_types.h"
#include "kernels.h"
#include "prim_common.cuh"

namespace gint {

// D = A B + D on the FP64 tensor cores: A 8 x 4 (lane: row lane / 4, column lane % 4), B 4 x 8 (row
// lane % 4, column lane / 4), D 8 x 8 (row lane / 4, columns 2 (lane % 4) and the next).
static __device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
   asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
       : "+d"(d0), "+d"(d1)
       : "d"(a), "d"(b));
}

// eight bytes from global to shared memory, without passing a register
static __device__ __forceinline__ void copy8_async(double *to, const double *from) {
   asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
static __device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr int kMmThreads = 256;    // the most threads of a block
constexpr int kMmPrims = 32;       // primitives whose coefficients are in shared memory at a time
constexpr int kMmCoefStride = 12;  // doubles from one to the next (conflict-free operand reads)
constexpr int kMmRootDoubles = 34; // HRR inputs that a lane keeps in registers; longer ones it rereads

__host__ __device__ constexpr int mm_nc(int l) { return (l + 1) * (l + 2) / 2; }
// cartesians of the shells l0..l1
__host__ __device__ constexpr int mm_sum(int l0, int l1) {
   int n = 0;
   for (int l = l0; l <= l1; l++) n += mm_nc(l);
   return n;
}
// Exponent y + z of a shell's i-th cartesian, the index of that cartesian times x, y or z, and the first
// axis with a nonzero exponent of the j-th cartesian of degree d (2 for d = 0).
__host__ __device__ constexpr int mm_yz(int i) { return (i >= 1) + (i >= 3) + (i >= 6) + (i >= 10) + (i >= 15); }
__host__ __device__ constexpr int mm_up(int i, int t) { return t == 0 ? i : i + mm_yz(i) + t; }
__host__ __device__ constexpr int mm_first(int d, int j) { return mm_yz(j) < d ? 0 : (j < d * (d + 1) / 2 + d ? 1 : 2); }

// f(m) for m < N, a template constant
template <class F, int... M>
static __device__ __forceinline__ void mm_for(const F &f, std::integer_sequence<int, M...>) { (f(std::integral_constant<int, M>()), ...); }
template <int N, class F>
static __device__ __forceinline__ void mm_for(const F &f) { mm_for(f, std::make_integer_sequence<int, N>()); }

// The HRR of one pair (l0 lb: node (D, J) holds the elements (l, J) of l = L0 .. L0 + LB - D for the
// J-th cartesian of degree D, and makes (l, J + 1_t) = (l + 1_t, J) + R_t (l, J) for the J + 1_t whose
// first axis is t. Depth first, so that one chain of nodes is live at a time; emit gets each (L0, J)
// of degree LB.
template <int L0, int LB, int D = 0, int J = 0>
struct Hrr {
   template <class H, class F>
   static __device__ __forceinline__ void run(const H &h, const double *R, const F &emit) {
      if constexpr (D == LB) {
         emit(std::integral_constant<int, J>(), h);
      } else {
         child<0>(h, R, emit);
         if constexpr (mm_first(D, J) >= 1) child<1>(h, R, emit);
         if constexpr (mm_first(D, J) >= 2) child<2>(h, R, emit);
      }
   }
   template <int T, class H, class F>
   static __device__ __forceinline__ void child(const H &h, const double *R, const F &emit) {
      double v[mm_sum(L0, L0 + LB - D - 1)];
      fill<T>(h, R, v, std::make_integer_sequence<int, mm_sum(L0, L0 + LB - D - 1)>());
      Hrr<L0, LB, D + 1, mm_up(J, T)>::run(v, R, emit);
   }
   // (the indices are template constants: unrolled loops over them took a minute to compile for f shells)
   template <int T, class H, int... I>
   static __device__ __forceinline__ void fill(const H &h, const double *R, double *v, std::integer_sequence<int, I...>) {
      ((v[I] = fma(R[T], h[I], h[std::integral_constant<int, raised(I, T)>::value])), ...);
   }
   // where the i-th element of the shells from L0 on, times axis t, is
   static __host__ __device__ constexpr int raised(int i, int t) {
      int l = L0;
      while (i >= mm_sum(L0, l)) l++;
      return mm_sum(L0, l) + mm_up(i - mm_sum(L0, l - 1), t);
   }
   // doubles that a lane holds at most
   static __host__ __device__ constexpr int live() {
      int n = mm_sum(L0, L0 + LB) <= kMmRootDoubles ? mm_sum(L0, L0 + LB) : 0;
      for (int d = 1; d <= LB; d++) n += mm_sum(L0, L0 + LB - d);
      return n;
   }
};

// every ST-th double of shared memory
template <int ST>
struct Strided {
   const double *p;
   __device__ __forceinline__ double operator[](int i) const { return p[i * ST]; }
};

// the HRR of one pair from N = ncart(l0..l0 + lb) inputs in shared memory
template <int L0, int LB, int ST, class F>
static __device__ __forceinline__ void mm_hrr(const double *in, const double *R, const F &emit) {
   constexpr int N = mm_sum(L0, L0 + LB);
   const Strided<ST> s{in};
   if constexpr (N <= kMmRootDoubles) {
      double h[N];
      mm_for<N>([&](auto i) { h[i.value] = s[i.value]; });
      Hrr<L0, LB>::run(h, R, emit);
   } else {
      Hrr<L0, LB>::run(s, R, emit);
   }
}

// spherical functions of one shell, [l][m][cartesian] (group_mm_preload)
__constant__ double c_mm_c2s[4][70];

// the m-th spherical function of a shell from its cartesians, zero coefficients left out
template <int L, int M, class X, int... K>
static __device__ __forceinline__ double mm_sph_sum(const X &x, std::integer_sequence<int, K...>) {
   double v = 0.0;
   auto add = [&](auto k) {
      if constexpr (c2s_mask(L, M) >> k.value & 1) v = fma(c_mm_c2s[L][M * mm_nc(L) + k.value], x[k.value], v);
   };
   (add(std::integral_constant<int, K>()), ...);
   return v;
}
template <int L, int M, class X>
static __device__ __forceinline__ double mm_sph(const X &x) {
   if constexpr (L == 0) return x[0];
   else return mm_sph_sum<L, M>(x, std::make_integer_sequence<int, mm_nc(L)>());
}
// Shapes of a class and its shared memory (doubles). One row: its targets T[f][e] (later its spherical
// integrals I), the ket's HRR X[cd][e], the cartesian sum C[ab][cd]; the strides are odd, so that
// lanes along e, along cd and along ab fall on different banks.
template <int CLS>
struct MmShape {
   static constexpr int LA = CLS >> 6, LB = CLS >> 4 & 3, LC = CLS >> 2 & 3, LD = CLS & 3;
   static constexpr int NA = 2 * LA + 1, NB = 2 * LB + 1, NC = 2 * LC + 1, ND = 2 * LD + 1, NCD = NC * ND;
   static constexpr int ncb = mm_nc(LB), ncc = mm_nc(LC), ncd = mm_nc(LD), nab = mm_nc(LA) * ncb, nkt = ncc * ncd;
   static constexpr int nE = mm_sum(LA, LA + LB), nF = mm_sum(LC, LC + LD), S = nE * nF;
   static constexpr int ES = nE | 1, CS = nkt | 1;
   static constexpr int oX = nF * ES, oC = oX + nkt * ES, row = (oC + nab * CS) | 1;
   static constexpr int nout = (NA + NB) * (NC + ND);
   // eight rows a tile (the height of a product), fewer where two blocks would not fit an SM
   static __host__ __device__ constexpr int rows() {
      for (int r = 8; r > 1; r /= 2)
         if ((kMmPrims * kMmCoefStride + r * (row + nout)) * 8 <= 112 * 1024) return r;
      return 1;
   }
   static constexpr int RT = rows();
   static constexpr bool kWide = RT < 4;   // a row is worked on by the block, else by one warp
   static constexpr int regs = 2 * (Hrr<LA, LB>::live() > Hrr<LC, LD>::live() ? Hrr<LA, LB>::live() : Hrr<LC, LD>::live()) + 40;
   static constexpr int MINB = regs <= 80 ? 3 : (regs <= 128 ? 2 : 1);
   static __host__ __device__ constexpr int doubles(int nspin) { return kMmPrims * kMmCoefStride + RT * (row + nspin * nout); }
};

// One row's P/K block of one pair (ac, ad, bc, bd): element (x, y) is at off + x sx + y sy.
struct MmBlock {
   uint32_t off;
   int sx, sy, ok;
};

// r / n for r < 256 and n in 1..4
static __device__ __forceinline__ int div_nl(int r, int n) {
   const unsigned m = n == 1 ? 65536u : (n == 2 ? 32768u : (n == 3 ? 21846u : 16384u));
   return (int)(((unsigned)r * m) >> 16);
}

// One block per group (all image pairs of one set quartet for one class); RT contraction rows at
// a time (blockIdx.y deals the tiles of a group out where there are few groups). Per shell quartet:
//  1. coefficient products of the rows and 32 primitives at a time;
//  2. T = coefficients x AC on the FP64 tensor cores, eight targets a tile, into shared memory;
//  3. lane per (row, e): the ket's HRR of T[.][e] in registers, into X;
//  4. lane per (row, cd): the bra's HRR of X[cd][.], added to C; after the last shell quartet also the
//     spherical transform of a and b;
// then, lane per (row, ab), that of c and d, and the K update of the rows, one thread per element of
// the four blocks. The lanes of stages 3 and 4 of one row are one warp (the block where a tile has one or
// two rows), so that no barrier of the block lies between them.
// What bounds it: chains of short stages between barriers, with loads of primitives and P at their heads.
// As dense products B T K with precomputed B and K, the HRR and transform of this kernel took five times the
// operations and up to seven eighths of them on the padding of tiles that shared memory had cut to 1, 2 or
// 4 rows. Group time of the classes of L = 4..6 and 7..11, kernels one after another, with the products and
// now: 27.3 and 20.0 ms, 12.4 and 7.5 ms on the 1/4096 sample of the 64-molecule l <= 3 workload; 3.6 and
// 2.6 ms, 4.2 and 2.4 ms on 24 clusters. (pp|pp) issues in 52 % of the cycles, its L1 data pipe is 48 % busy,
// and of 8 warps a scheduler could hold 5 are there, mostly at a barrier (2.7 per issued instruction).
template <int CLS>
__global__ void __launch_bounds__(kMmThreads, MmShape<CLS>::MINB) k_group_mm(DevCtx ctx, BatchArgs bt) {
   using Sh = MmShape<CLS>;
   constexpr int NA = Sh::NA, NB = Sh::NB, NC = Sh::NC, ND = Sh::ND, NCD = Sh::NCD, S = Sh::S, RT = Sh::RT, ROW = Sh::row;
   constexpr int ES = Sh::ES, CS = Sh::CS, ncb = Sh::ncb, nout = Sh::nout;
   extern __shared__ __align__(16) double smem[];
   __shared__ double shell_vec[2][6];
   __shared__ MmBlock blk[8][4];
   __shared__ double row_fac[8];
   double *cw = smem, *rows = smem + kMmPrims * kMmCoefStride, *Pm = rows + RT * ROW;
   const int tid = threadIdx.x, nth = blockDim.x, warp = tid >> 5, lane = tid & 31, nw = nth >> 5;
   const int lr = lane >> 2, lq = lane & 3;
   // this thread's element of the four K blocks in the K update: block u, its place (x, y), the bra and
   // ket functions summed over (nx2, ny2) and the strides in I; threads beyond rpp * nout have none
   const int rpp = max(1, nth / nout), orow = tid / nout;
   auto element = [&](int o, int &u, int &x, int &y, int &nx2, int &ny2, int &at, int &sx2, int &sy2) {
      constexpr int na = NA * (NC + ND);
      const bool bra_b = o >= na;
      if (bra_b) o -= na;
      const int nx = bra_b ? NB : NA;
      const bool ket_d = o >= nx * NC;
      if (ket_d) o -= nx * NC;
      const int ny = ket_d ? ND : NC;
      x = o / ny; y = o - x * ny;
      u = (bra_b ? 2 : 0) + (ket_d ? 1 : 0);
      nx2 = bra_b ? NA : NB; ny2 = ket_d ? NC : ND;
      at = x * (bra_b ? NCD : NB * NCD) + y * (ket_d ? 1 : ND);
      sx2 = bra_b ? NB * NCD : NCD; sy2 = ket_d ? ND : 1;
   };
   // where target j (a panel [nE][ncart(f)] per ket shell f) goes in T
   auto place = [](int j) {
      int at = 0;
#pragma unroll
      for (int f = Sh::LC; f <= Sh::LC + Sh::LD; f++) {
         const int f0 = mm_sum(Sh::LC, f - 1), i = j - f0 * Sh::nE, e = i / mm_nc(f);
         if (i >= 0) at = (f0 + i - e * mm_nc(f)) * ES + e;
      }
      return at;
   };
   // f(row, i) for i < n of the tile's nr rows: those of a row by the lanes of its warp, or by the block
   auto each = [&](int nr, int n, auto f) {
      if constexpr (Sh::kWide) {
         for (int i = tid; i < nr * n; i += nth) f(i / n, i % n);
      } else {
         const int rpw = (nr + nw - 1) / nw, w0 = warp * rpw, mine = max(0, min(rpw, nr - w0)) * n;
         for (int i = lane; i < mine; i += 32) f(w0 + i / n, i % n);
      }
   };
   auto each_done = [] {
      if constexpr (Sh::kWide) __syncthreads();
      else __syncwarp();
   };

   for (uint32_t g = blockIdx.x; g < bt.ngroup; g += gridDim.x) {
      if (bt.gflags && !__ldg(bt.gflags + g)) continue;   // screened on an incremental replay
      const GroupRec G = bt.groups[g];
      const int n1 = G.nl[1], n2 = G.nl[2], n3 = G.nl[3], nrow = G.nl[0] * n1 * n2 * n3;
      for (int r0 = blockIdx.y * RT; r0 < nrow; r0 += gridDim.y * RT) {
         const int nr = min(RT, nrow - r0);
         __syncthreads();                                  // the previous tile is done with all of it
         if (tid < 4 * nr) {
            const QrttRec k = bt.qrtts[G.qrtt_off + r0 + (tid >> 2)];
            const int u = tid & 3;
            const bool T = (k.T >> u) & 1, ok = row_in_range(k, NA, NB, NC, ND, ctx.FP_size);
            blk[tid >> 2][u] = {k.off[u], T ? (int)k.ld[u] : 1, T ? 1 : (int)k.ld[u], ok ? 1 : 0};
            if (u == 0) row_fac[tid >> 2] = -ctx.hf_fac * (k.idx_fac == 4 ? 0.0 : 2.0 / (double)(1 << k.idx_fac));
            if (!ok) atomicOr(ctx.err, 1);
         }
         // the contraction of this thread's row in the coefficient products
         const int cr = tid & 7, r = r0 + min(cr, nr - 1);
         const int rd = div_nl(r, n3), rc = div_nl(rd, n2), ia = div_nl(rc, n1);
         const int ib = rc - ia * n1, ic = rd - rc * n2, id = r - rd * n3;
         for (uint32_t s = 0; s < G.nshell; s++) {
            const ShellRec sh = bt.shells[G.shell_off + s];
            const BasisEnt &ea = ctx.ents[sh.ent[0]], &eb = ctx.ents[sh.ent[1]];
            const BasisEnt &ec = ctx.ents[sh.ent[2]], &ed = ctx.ents[sh.ent[3]];
            const double *Ka = ctx.pool + ea.k_off + ia * ea.np, *Kb = ctx.pool + eb.k_off + ib * eb.np;
            const double *Kc = ctx.pool + ec.k_off + ic * ec.np, *Kd = ctx.pool + ed.k_off + id * ed.np;
            double *vec = shell_vec[s & 1];   // A - B, C - D: the other shells' lanes may still read theirs
            if (tid == 0) read_shell_vectors(ctx, bt, G.shell_off + s, sh, vec);
            for (uint32_t p0 = 0; p0 < sh.nprm || p0 == 0; p0 += kMmPrims) {
               const int np = (int)min((uint32_t)kMmPrims, sh.nprm - p0), npp = (np + 3) & ~3;
               for (int p = tid >> 3; p < npp; p += nth >> 3) {
                  double v = 0.0;
                  if (p < np && cr < nr) {
                     const uint32_t code = __ldg(bt.prm + sh.prm_off + p0 + p);
                     v = __ldg(Ka + (code >> 24)) * __ldg(Kb + ((code >> 16) & 255)) * __ldg(Kc + ((code >> 8) & 255)) *
                         __ldg(Kd + (code & 255));
                  }
                  cw[p * kMmCoefStride + cr] = v;
               }
               // the targets of the warp's first tile and first eight primitives are on their way meanwhile
               const double *ac = bt.AC + (size_t)(sh.prm_off + p0) * S;
               auto target = [&](int p, int j) { return p < np && j < S ? __ldg(ac + (size_t)p * S + j) : 0.0; };
               double b0[2][2];
#pragma unroll
               for (int q = 0; q < 2; q++)
#pragma unroll
                  for (int t = 0; t < 2; t++) b0[q][t] = target(lq + 4 * q, warp * 16 + lr + 8 * t);
               __syncthreads();
               if (s == 0 && p0 == 0) {
                  // P's elements of the rows, in the order of the K update's elements
                  for (int i = tid; i < nr * nout; i += nth) {
                     const int row = i / nout, o = i - row * nout;
                     int u, x, y, nx2, ny2, at, sx2, sy2;
                     element(o, u, x, y, nx2, ny2, at, sx2, sy2);
                     const MmBlock b = blk[row][u];
                     if (b.ok)
                        for (int sp = 0; sp < ctx.nspin; sp++)
                           copy8_async(Pm + (sp * RT + row) * nout + o, ctx.P[sp] + ((size_t)b.off + x * b.sx + y * b.sy));
                  }
               }
               // T of 16 targets a warp at a time, on from the sums of the primitives before
               for (int j0 = warp * 16; j0 < S; j0 += nw * 16) {
                  double t[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
                  double *at[4];
#pragma unroll
                  for (int u = 0; u < 4; u++) {
                     const int j = j0 + 2 * lq + (u & 1) + (u >> 1) * 8;
                     at[u] = lr < nr && j < S ? rows + lr * ROW + place(j) : nullptr;
                     if (p0 && at[u]) t[u >> 1][u & 1] = *at[u];
                  }
#pragma unroll
                  for (int q = 0; q < 2; q++) {
                     if (4 * q >= npp) break;
                     const double a = cw[(lq + 4 * q) * kMmCoefStride + lr];
                     dmma(t[0][0], t[0][1], a, b0[q][0]);
                     dmma(t[1][0], t[1][1], a, b0[q][1]);
                  }
#pragma unroll 4
                  for (int p = lq + 8; p < npp; p += 4) {
                     const double a = cw[p * kMmCoefStride + lr];
                     const double ba = target(p, j0 + lr), bb = target(p, j0 + lr + 8);
                     dmma(t[0][0], t[0][1], a, ba);
                     dmma(t[1][0], t[1][1], a, bb);
                  }
#pragma unroll
                  for (int q = 0; q < 2; q++)
#pragma unroll
                     for (int u = 0; u < 2; u++) b0[q][u] = target(lq + 4 * q, j0 + nw * 16 + lr + 8 * u);
#pragma unroll
                  for (int u = 0; u < 4; u++)
                     if (at[u]) *at[u] = t[u >> 1][u & 1];
               }
               __syncthreads();
            }
            // the ket's HRR
            {
               const double R[3] = {vec[3], vec[4], vec[5]};
               each(nr, Sh::nE, [&](int row, int e) {
                  double *x = rows + row * ROW + Sh::oX + e;
                  mm_hrr<Sh::LC, Sh::LD, ES>(rows + row * ROW + e, R, [&](auto J, const auto &v) {
                     mm_for<Sh::ncc>([&](auto c) { x[(c.value * Sh::ncd + J.value) * ES] = v[c.value]; });
                  });
               });
            }
            each_done();
            // the bra's HRR, the sum of the shell quartets, and the transform of a and b
            {
               const double R[3] = {vec[0], vec[1], vec[2]};
               const bool first = s == 0, last = s + 1 == G.nshell;
               each(nr, Sh::nkt, [&](int row, int cd) {
                  double *C = rows + row * ROW + Sh::oC + cd;   // [ab], stride CS
                  mm_hrr<Sh::LA, Sh::LB, 1>(rows + row * ROW + Sh::oX + cd * ES, R, [&](auto J, const auto &v) {
                     constexpr int nca = mm_nc(Sh::LA);
                     double sum[nca];
                     mm_for<nca>([&](auto a) { sum[a.value] = first ? v[a.value] : C[(a.value * ncb + J.value) * CS] + v[a.value]; });
                     if (last) mm_for<NA>([&](auto a) { C[(a.value * ncb + J.value) * CS] = mm_sph<Sh::LA, a.value>(sum); });
                     else mm_for<nca>([&](auto a) { C[(a.value * ncb + J.value) * CS] = sum[a.value]; });
                  });
                  if (Sh::LB > 0 && last) {
                     // in place: function (a, b) goes where cartesians up to those of a were
                     mm_for<NA>([&](auto a) {
                        double x[ncb];
                        mm_for<ncb>([&](auto b) { x[b.value] = C[(a.value * ncb + b.value) * CS]; });
                        mm_for<NB>([&](auto b) { C[(a.value * NB + b.value) * CS] = mm_sph<Sh::LB, b.value>(x); });
                     });
                  }
               });
            }
         }
         if (G.nshell == 0) continue;
         each_done();
         // the transform of c and d, into T's place
         each(nr, NA * NB, [&](int row, int ab) {
            const double *C = rows + row * ROW + Sh::oC + ab * CS;
            double *I = rows + row * ROW + ab * NCD;
            mm_for<NC>([&](auto c) {
               double x[Sh::ncd];
               mm_for<Sh::ncd>([&](auto d) { x[d.value] = mm_sph<Sh::LC, c.value>(Strided<Sh::ncd>{C + d.value}); });
               mm_for<ND>([&](auto d) { I[c.value * ND + d.value] = mm_sph<Sh::LD, d.value>(x); });
            });
         });
         copies_done();
         __syncthreads();
         // K update (reference src/compute_KS.cpp:26-115): element (x, y) of one of the blocks ac, ad,
         // bc, bd gets minus the sum over the other bra and ket function of I times the P of their block
         for (int o0 = 0; o0 < nout; o0 += nth) {   // one round unless a row has more elements than threads
            const int o = rpp > 1 ? tid - orow * nout : o0 + tid;
            if (o >= nout || orow >= rpp) continue;
            int u, x, y, nx2, ny2, at, sx2, sy2;
            element(o, u, x, y, nx2, ny2, at, sx2, sy2);
            // where the partner block 3 - u starts among the elements
            const int pu = 3 - u, pb = (pu & 2 ? NA * (NC + ND) : 0) + (pu & 1 ? (pu & 2 ? NB : NA) * NC : 0);
            for (int row = rpp > 1 ? orow : 0; row < nr; row += rpp) {
               const MmBlock to = blk[row][u];
               if (!to.ok) continue;
               const double *I = rows + row * ROW + at, f = row_fac[row];
               for (int sp = 0; sp < ctx.nspin; sp++) {
                  const double *P = Pm + (sp * RT + row) * nout + pb;
                  double v = 0.0;
                  for (int i = 0; i < nx2; i++) {
#pragma unroll 3
                     for (int j = 0; j < ny2; j++) v += I[i * sx2 + j * sy2] * P[i * ny2 + j];
                  }
                  atomicAdd(ctx.K[sp] + ((size_t)to.off + x * to.sx + y * to.sy), f * v);
               }
            }
         }
      }
   }
}

}  // namespace gint
