// kernels.cu -- sm_100a kernels of the K build.
//
// Two kernels per angular-momentum class (la,lb,lc,ld), launched on class-sorted segments of
// one batch:
//
//  k_prim3, k_prim2   the image-summed (e0|f0)^(0) targets of every primitive quartet, into the AC
//               buffer: truncated-Coulomb G_m by the patch Chebyshev series or the Boys function
//               for the images that pass the truncation test, then the Obara-Saika VRR of each
//               surviving image, generated per lane (prim3.cu) or interpreted by a team (below).
//               (reference: src/compute_Fm.cpp:20-326, src/compute_VRR.cpp:349-458,
//                src/compute_ECO.cpp:216-272)
//  k_group3, k_group_mm, k_group   for every contraction row of every group (all image pairs of one set
//               quartet), contract AC over the primitives of each shell, apply the HRR with that
//               shell's AB/CD, sum the shells, transform to spherical and update K with atomics:
//               one lane per row (group3.cu), one block per group (group_mm.cuh), or one warp per
//               row (below).
//               (reference: src/compute_ECO.cpp:12-214, src/compute_HRR.cpp:102-225,
//                src/compute_SPH.cpp:58-237, src/compute_KS.cpp:8-117)
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include "engine_types.h"
#include "kernels.h"
#include "group3.h"
#include "group_mm.h"
#include "prim3.h"
#include "prim_common.cuh"

namespace gint {

__constant__ double c_c2s[4][70];
__constant__ double c_symm[5];

static __device__ __forceinline__ int ncart(int l) { return (l + 1) * (l + 2) / 2; }

// ---------------------------------------------------------------------------------------
// k_prim2<NT>: Fm + VRR + sum over n3 for the classes without generated VRR code. One team of NT
// threads (a warp, or a whole block) per chunk of primitive quartets:
//  1. lane per primitive of the chunk: its geometry into shared memory;
//  2. lane per (primitive, image) pair, over the images short enough to pass: the truncation test;
//     passing pairs queue up in primitive order, and a batch of 32 (or the chunk's rest) goes on;
//  3. lane per queued pair, the warps of the team sharing its orders: G_m (Chebyshev or Boys);
//  4. the team, image after image with Fm[0] > 1e-12: the VRR as one precompiled instruction per
//     element, level by level, and the m = 0 targets stored to (the first image of a primitive) or
//     added to the primitive's row in AC, always by the same thread.
// What bounds it: chains of dependent loads and FP64 operations, a batch or an image after another.
// Chunks of up to 16 primitives fill the lanes of stages 1 to 3 (a chunk sized by the accumulators
// of its targets held one or two primitives, and G_m ran with 3 lanes of 32); adding to AC in
// place leaves shared memory to the workspace, so more teams are resident; each thread loads its
// next instruction before it runs the present one. The classes of L >= 5 of the 1/4096 sample of
// the 64-molecule l <= 3 workload: 27.4 ms before, 16.7 ms now; 2 molecules, 27 images, 27k
// primitive quartets over 250 classes: 25.2 to 12.1 ms, kernels one after another.
// ---------------------------------------------------------------------------------------
constexpr int kPrim2Chunk = 16;

// the barrier of one team of NT threads
template <int NT>
static __device__ __forceinline__ void tsync() {
   if constexpr (NT > 32) __syncthreads();
   else __syncwarp();
}

template <int NT>
__global__ void __launch_bounds__(NT == 32 ? 256 : NT, NT == 32 ? 2 : (NT == 128 ? 4 : 1))
k_prim2(DevCtx ctx, BatchArgs bt, int cp, int team_doubles) {
   extern __shared__ __align__(16) double smem[];
   write_shell_vectors(ctx, bt);
   ClassPlan *pl = reinterpret_cast<ClassPlan *>(smem);
   {
      const int nwords = (int)(sizeof(ClassPlan) / 4);
      const int *src = reinterpret_cast<const int *>(bt.plan);
      int *dst = reinterpret_cast<int *>(smem);
      for (int w = threadIdx.x; w < nwords; w += blockDim.x) dst[w] = src[w];
   }
   __syncthreads();
   const int plan_doubles = (int)((sizeof(ClassPlan) + 15) / 16) * 2;
   const int team = threadIdx.x / NT, tl = threadIdx.x % NT, lane = threadIdx.x & 31, tw = tl >> 5;
   const int nteam = blockDim.x / NT;
   double *tb = smem + plan_doubles + (size_t)team * team_doubles;
   const int L = pl->L, S = pl->S, Ng = ctx.Ng, LF = L + 1;
   // per-team layout (prim2_team_doubles)
   PrimGeo *geo = reinterpret_cast<PrimGeo *>(tb);                     // [cp]
   double *s00 = tb + cp * (int)(sizeof(PrimGeo) / 8);                 // [cp]
   double *q1t = s00 + cp;                                            // [64] T of the queued pairs
   int *q1i = reinterpret_cast<int *>(q1t + 64);                      // [64] primitive << 8 | image
   double *q2f = q1t + 64 + 32;                                       // [32][LF] Fm of the batch
   double *pqz = q2f + 32 * LF;                                       // [18] factors of one image
   double *ws = pqz + 18;                                             // [V] VRR workspace and a zero
   const bool want00 = pl->want00 != 0, need_vrr = !(want00 && pl->ntg == 1);
   const int s00_at = want00 ? pl->s00 : -1;
   const unsigned below = (1u << lane) - 1u;
   const int4 *vop = reinterpret_cast<const int4 *>(ctx.vops + pl->vop_off);
   const uint16_t *tmap = ctx.tmap + pl->tmap_off;
   const int nvop = pl->nvop, nlev = pl->nlev;
   unsigned long long c_cheb = 0, c_boys = 0, c_vrr = 0;
   if (tl == 0) ws[pl->V] = 0.0;

   const uint32_t nchunk = (bt.nprm + cp - 1) / cp;
   for (uint32_t ch = blockIdx.x * nteam + team; ch < nchunk; ch += gridDim.x * nteam) {
      const uint32_t p0 = ch * cp;
      const int np = (int)min((uint32_t)cp, bt.nprm - p0);
      // every warp of the team numbers and tests the pairs for itself, from the geometry of warp 0
      tsync<NT>();
      if (tw == 0 && lane < np) {
         PrimGeo g;
         const ShellRec sh = bt.shells[bt.prm_shell[p0 + lane]];
         prim_geometry(ctx, sh, bt.prm[p0 + lane], g);
         kill_if_screened(bt, sh, g);
         geo[lane] = g;
         s00[lane] = 0.0;
      }
      tsync<NT>();
      int start;
      const int nimg = lane < np ? image_count(ctx.img, Ng, geo[lane]) : 0;
      const int npair = pair_starts(nimg, np, lane, start);
      double *out = bt.AC + (size_t)p0 * S;
      unsigned done = 0;   // primitives whose row holds an image already
      // stages 3 and 4 of the queued pairs [0, cnt)
      auto run_batch = [&](int cnt) {
         if (lane < cnt) {
            const int pk = q1i[lane];
            const int br = fm_eval_geo<-1>(ctx, L, geo[pk >> 8], q1t[lane], q2f + lane * LF, tw, NT / 32);
            if (tw == 0) { c_cheb += (br == 1); c_boys += (br == 2); }
         }
         tsync<NT>();
         const double f0 = lane < cnt ? q2f[lane * LF] : 0.0;
         if (want00 && tw == 0) {
            const int p = lane < cnt ? q1i[lane] >> 8 : -1 - lane;
            SegSum<double> sg = make_segsum<double>(p, lane, s00 + max(p, 0));
            sg(0, f0);
         }
         unsigned bal = __ballot_sync(0xffffffffu, need_vrr && lane < cnt && f0 > 1.e-12);
         if (tl == 0) c_vrr += __popc(bal);
         for (; bal; bal &= bal - 1) {
            const int s = __ffs(bal) - 1, pk = q1i[s], p = pk >> 8;
            const PrimGeo &g = geo[p];
            if (tl < 3) {
               const double Qp = g.Q[tl] + __ldg(reinterpret_cast<const double *>(ctx.img + (pk & 255)) + tl);
               const double W = wdist(g.zab, g.P[tl], g.zcd, Qp, g.inv_z);
               pqz[tl] = g.PA[tl]; pqz[3 + tl] = W - g.P[tl]; pqz[6 + tl] = g.QC[tl]; pqz[9 + tl] = W - Qp;
            } else if (tl == 3) {
               pqz[12] = g.i2ab; pqz[13] = g.mrab; pqz[14] = g.i2cd; pqz[15] = g.mrcd; pqz[16] = g.i2z;
            }
            if (tl < LF) ws[tl] = q2f[s * LF + tl];   // (0|0)^(m), m = 0..L
            int4 next = __ldg(vop + min(tl, nvop - 1));
            tsync<NT>();
            int e0 = 0;
            for (int lv = 1; lv <= nlev; lv++) {
               const int e1 = pl->vop_lev[lv];
               for (int e = e0 + tl; e < e1; e += NT) {
                  VOp o;
                  memcpy(&o, &next, sizeof(VOp));
                  const int en = e + NT < e1 ? e + NT : e1 + tl;
                  next = __ldg(vop + min(en, nvop - 1));
                  double v = pqz[o.zA] * ws[o.i0] + pqz[o.zA + 3] * ws[o.i1];
                  if (o.f1) v += o.f1 * (pqz[12 + 2 * o.kind] * ws[o.i2] + pqz[13 + 2 * o.kind] * ws[o.i3]);
                  if (o.f2) v += o.f2 * pqz[16] * ws[o.i4];
                  ws[o.out] = v;
               }
               if (e0 + tl >= e1) next = __ldg(vop + min(e1 + tl, nvop - 1));   // idle on this level
               e0 = e1;
               tsync<NT>();
            }
            double *row = out + (size_t)p * S;
            if (done >> p & 1) {
               for (int j = tl; j < S; j += NT)
                  if (j != s00_at) row[j] += ws[__ldg(tmap + j)];
            } else {
               for (int j = tl; j < S; j += NT)
                  if (j != s00_at) row[j] = ws[__ldg(tmap + j)];
            }
            done |= 1u << p;
            tsync<NT>();
         }
      };
      // stage 2
      int n1 = 0;
      for (int b0 = 0; b0 < npair; b0 += 32) {
         bool pass = false;
         double T = 0.0;
         int tn;
         const int tp = pair_prim(ctx, b0, npair, start, nimg, lane, tn);
         if (b0 + lane < npair) {
            const PrimGeo &g = geo[tp];
            const double *im = reinterpret_cast<const double *>(ctx.img + tn);
            const double d0 = rsub(g.D[0], __ldg(im)), d1 = rsub(g.D[1], __ldg(im + 1)), d2 = rsub(g.D[2], __ldg(im + 2));
            T = rmul(g.rho, rdot3(d0, d0, d1, d1, d2, d2));
            pass = !(T > g.upper);
         }
         const unsigned bal = __ballot_sync(0xffffffffu, pass);
         if (pass && tw == 0) {
            const int pos = n1 + __popc(bal & below);
            q1i[pos] = (tp << 8) | tn;
            q1t[pos] = T;
         }
         n1 += __popc(bal);
         tsync<NT>();
         if (n1 >= 32) {
            run_batch(32);
            const int rem = n1 - 32;
            int vi = 0;
            double vt = 0.0;
            tsync<NT>();
            if (tw == 0 && lane < rem) { vi = q1i[32 + lane]; vt = q1t[32 + lane]; }
            tsync<NT>();
            if (tw == 0 && lane < rem) { q1i[lane] = vi; q1t[lane] = vt; }
            tsync<NT>();
            n1 = rem;
         }
      }
      if (n1 > 0) run_batch(n1);
      // the rows without an image, and the (00|00) target, which collects every image's Fm[0]
      // (reference src/compute_VRR.cpp:381-389)
      tsync<NT>();
      for (int p = 0; p < np; p++)
         if (!(done >> p & 1))
            for (int j = tl; j < S; j += NT)
               if (j != s00_at) out[(size_t)p * S + j] = 0.0;
      if (want00 && tl < np) out[(size_t)tl * S + s00_at] = s00[tl];
      if (tl == 0 && ctx.cnt) atomicAdd(ctx.cnt + bt.cls * 4 + 3, (unsigned long long)np);
   }
   if (ctx.cnt && tw == 0) {
      for (int o = 16; o > 0; o >>= 1) {
         c_cheb += __shfl_down_sync(0xffffffffu, c_cheb, o);
         c_boys += __shfl_down_sync(0xffffffffu, c_boys, o);
      }
      if (lane == 0) {
         atomicAdd(ctx.cnt + bt.cls * 4 + 0, c_cheb);
         atomicAdd(ctx.cnt + bt.cls * 4 + 1, c_boys);
         atomicAdd(ctx.cnt + bt.cls * 4 + 2, c_vrr);
      }
   }
}

// ---------------------------------------------------------------------------------------
// k_group: contraction + HRR + sum over image pairs + spherical transform + K update
// ---------------------------------------------------------------------------------------
// One spherical pass over centre LX: the workspace is [npre][ncart(LX)][npost] in, and
// [npre][2LX+1][npost] out. Each lane transforms whole vectors (one (pre, post) pair at a time),
// so the coefficients are uniform across the warp. Same sum order as a dense row loop.
template <int LX>
static __device__ __forceinline__ void sph_pass(const double *src, double *dst, int npre, int npost, int lane) {
   constexpr int NK = (LX + 1) * (LX + 2) / 2, NSX = 2 * LX + 1;
   const int nu = npre * npost;
   for (int u = lane; u < nu; u += 32) {
      const int pre = u / npost, post = u - pre * npost;
      const double *s = src + pre * NK * npost + post;
      double *d = dst + pre * NSX * npost + post;
      double x[NK];
#pragma unroll
      for (int k = 0; k < NK; k++) x[k] = s[k * npost];
#pragma unroll
      for (int m = 0; m < NSX; m++) {
         double acc = 0.0;
#pragma unroll
         for (int k = 0; k < NK; k++)
            if (c2s_mask(LX, m) >> k & 1) acc += c_c2s[LX][m * NK + k] * x[k];
         d[m * npost] = acc;
      }
   }
}

// q = t / n for t * n < 2^20, with M = 2^20 / n + 1 (all spherical indices here: t < 7^4, n <= 7^3)
static __device__ __forceinline__ int div_small(int t, uint32_t M) { return (int)(((uint32_t)t * M) >> 20); }

// What the rows of one set quartet share for one shell quartet: its primitive range, the
// coefficient rows of its four basis entries and the HRR displacements AB = A - B, CD = C - D.
struct ShellShared {
   uint32_t key;              // group index it was derived for (shell 0 of that group); ~0u: empty
   uint32_t prm_off, nprm;
   int k_off[4], np[4];
   double AB[3], CD[3];
};
static_assert(sizeof(ShellShared) <= kGroupShellCacheDoubles * 8, "shell cache slot too small");

static __device__ __forceinline__ void shell_shared(const DevCtx &ctx, const BatchArgs &bt, uint32_t i, ShellShared &o) {
   const ShellRec sh = bt.shells[i];
   o.prm_off = sh.prm_off; o.nprm = sh.nprm;
   for (int q = 0; q < 4; q++) {
      const BasisEnt &e = ctx.ents[sh.ent[q]];
      o.k_off[q] = e.k_off; o.np[q] = e.np;
   }
   double v[6];
   read_shell_vectors(ctx, bt, i, sh, v);
   for (int c = 0; c < 3; c++) { o.AB[c] = v[c]; o.CD[c] = v[3 + c]; }
}

// One contraction row q (of group gi = G) processed by one warp with workspace ws. In the cache slot
// (the warp's shared memory, key ~0u at first) shell 0's shared data is derived once and reused by the
// next rows of the same group that this warp takes.
static __device__ __forceinline__ void group_body(const DevCtx &ctx, const BatchArgs &bt, const ClassPlan *pl,
                                                  const GroupRec &G, uint32_t q, double *ws, double *cart, int lane,
                                                  const uint2 *hrec, double *kpw, ShellShared *cache, uint32_t gi) {
   const int S = pl->S, Nc = pl->Nc, Ns = pl->Ns;
   const int la = pl->la, lb = pl->lb, lc = pl->lc, ld = pl->ld;
   const int nca = ncart(la), ncb = ncart(lb), ncc = ncart(lc), ncd_ = ncart(ld);
   const int nsa = 2 * la + 1, nsb = 2 * lb + 1, nsc = 2 * lc + 1, nsd = 2 * ld + 1;
   const int nl1 = G.nl[1], nl2 = G.nl[2], nl3 = G.nl[3];
   {
      const int r = (int)(q - G.qrtt_off);
      const int ia = r / (nl1 * nl2 * nl3), ib = (r / (nl2 * nl3)) % nl1, ic = (r / nl3) % nl2, id = r % nl3;
      for (int x = lane; x < Nc; x += 32) cart[x] = 0.0;
      for (uint32_t s = 0; s < G.nshell; s++) {
         ShellShared sh;
         if (s == 0 && cache->key == gi) {
            sh = *cache;
         } else {
            shell_shared(ctx, bt, G.shell_off + s, sh);
            if (s == 0) {
               __syncwarp();
               if (lane == 0) { *cache = sh; cache->key = gi; }
               __syncwarp();
            }
         }
         const double *Ka = ctx.pool + sh.k_off[0] + ia * sh.np[0];
         const double *Kb = ctx.pool + sh.k_off[1] + ib * sh.np[1];
         const double *Kc = ctx.pool + sh.k_off[2] + ic * sh.np[2];
         const double *Kd = ctx.pool + sh.k_off[3] + id * sh.np[3];
         // contraction over primitives (reference src/compute_ECO.cpp:131-212)
         // the contraction coefficients of 32 primitives at a time, one per lane, then every
         // lane sums its targets over them in primitive order
         if (sh.nprm == 0)
            for (int j = lane; j < S; j += 32) ws[j] = 0.0;
         for (uint32_t p0 = 0; p0 < sh.nprm; p0 += 32) {
            const int np = (int)min(32u, sh.nprm - p0);
            if (lane < np) {
               const uint32_t code = __ldg(bt.prm + sh.prm_off + p0 + lane);
               kpw[lane] = __ldg(Ka + (code >> 24)) * __ldg(Kb + ((code >> 16) & 255)) *
                           __ldg(Kc + ((code >> 8) & 255)) * __ldg(Kd + (code & 255));
            }
            __syncwarp();
            const double *acp = bt.AC + (size_t)(sh.prm_off + p0) * S;
            for (int j = lane; j < S; j += 32) {
               double a = p0 ? ws[j] : 0.0;
               const double *rp = acp + j;
               int q = 0;
               for (; q + 4 <= np; q += 4) {
                  const double v0 = __ldg(rp), v1 = __ldg(rp + S), v2 = __ldg(rp + 2 * S), v3 = __ldg(rp + 3 * S);
                  a += kpw[q] * v0;
                  a += kpw[q + 1] * v1;
                  a += kpw[q + 2] * v2;
                  a += kpw[q + 3] * v3;
                  rp += 4 * S;
               }
               for (; q < np; q++) { a += kpw[q] * __ldg(rp); rp += S; }
               ws[j] = a;
            }
            __syncwarp();
         }
         __syncwarp();
         // HRR (reference src/compute_HRR.cpp:7-99), one precompiled instruction per element; the
         // elements of one level are independent, so each lane loads four before it stores any
         for (int lv = 1; lv <= pl->nhlev; lv++) {
            const HOp h0 = pl->hop[pl->hlev_off[lv - 1]], h1 = pl->hop[pl->hlev_off[lv] - 1];
            const int x0 = h0.out, x1 = h1.out + h1.nelem;
            double R0, R1, R2;
            if (h0.type == 0) { R0 = sh.CD[0]; R1 = sh.CD[1]; R2 = sh.CD[2]; }
            else { R0 = sh.AB[0]; R1 = sh.AB[1]; R2 = sh.AB[2]; }
            for (int x = x0 + lane; x < x1; x += 4 * 32) {
               uint2 ins[4];
#pragma unroll
               for (int u = 0; u < 4; u++) ins[u] = __ldg(&hrec[min(x + u * 32, x1 - 1) - S]);
               double w1[4], w2[4];
#pragma unroll
               for (int u = 0; u < 4; u++) { w1[u] = ws[ins[u].x & 0x3fffffffu]; w2[u] = ws[ins[u].y]; }
#pragma unroll
               for (int u = 0; u < 4; u++) {
                  if (x + u * 32 < x1) {
                     const uint32_t dir = ins[u].x >> 30;
                     const double Rd = dir == 0 ? R0 : (dir == 1 ? R1 : R2);
                     ws[x + u * 32] = w1[u] + Rd * w2[u];
                  }
               }
            }
            __syncwarp();
         }
         for (int x = lane; x < Nc; x += 32) cart[x] += ws[pl->out_off + x];
         __syncwarp();
      }
      // cartesian -> spherical, one centre at a time (a, b, c, d); the two halves of the
      // workspace take turns as the output, and l = 0 centres (a coefficient of 1) are skipped
      const double *sph = cart;
      {
         int dims[4] = {nca, ncb, ncc, ncd_};
         const int ls[4] = {la, lb, lc, ld};
         const int ns[4] = {nsa, nsb, nsc, nsd};
         for (int ctr = 0; ctr < 4; ctr++) {
            if (ls[ctr] == 0) continue;
            double *dst = (sph == ws) ? ws + Nc : ws;
            int npre = 1, npost = 1;
            for (int q = 0; q < ctr; q++) npre *= dims[q];
            for (int q = ctr + 1; q < 4; q++) npost *= dims[q];
            if (ls[ctr] == 1) sph_pass<1>(sph, dst, npre, npost, lane);
            else if (ls[ctr] == 2) sph_pass<2>(sph, dst, npre, npost, lane);
            else sph_pass<3>(sph, dst, npre, npost, lane);
            __syncwarp();
            dims[ctr] = ns[ctr];
            sph = dst;
         }
      }
      // K update (reference src/compute_KS.cpp:26-115)
      const QrttRec k = bt.qrtts[q];
      const double fac = c_symm[k.idx_fac] * ctx.hf_fac;
      const int nscd = nsc * nsd, nsbcd = nsb * nscd;
      const uint32_t Mbcd = (1u << 20) / nsbcd + 1, Mcd = (1u << 20) / nscd + 1, Md = (1u << 20) / nsd + 1;
      for (int t = lane; t < Ns; t += 32) {
         const int isa = div_small(t, Mbcd);
         int rem = t - isa * nsbcd;
         const int isb = div_small(rem, Mcd);
         rem -= isb * nscd;
         const int isc = div_small(rem, Md), isd = rem - isc * nsd;
         const int iac = !(k.T & 1) ? isc * k.ld[0] + isa : isa * k.ld[0] + isc;
         const int iad = !(k.T & 2) ? isd * k.ld[1] + isa : isa * k.ld[1] + isd;
         const int ibc = !(k.T & 4) ? isc * k.ld[2] + isb : isb * k.ld[2] + isc;
         const int ibd = !(k.T & 8) ? isd * k.ld[3] + isb : isb * k.ld[3] + isd;
         const size_t Iac = (size_t)k.off[0] + iac, Iad = (size_t)k.off[1] + iad;
         const size_t Ibc = (size_t)k.off[2] + ibc, Ibd = (size_t)k.off[3] + ibd;
         if (Iac >= ctx.FP_size || Iad >= ctx.FP_size || Ibc >= ctx.FP_size || Ibd >= ctx.FP_size) {
            atomicOr(ctx.err, 1);
            continue;
         }
         const double iabcd = -fac * sph[t];
         for (int sp = 0; sp < ctx.nspin; sp++) {
            const double *Pm = ctx.P[sp];
            double *Km = ctx.K[sp];
            atomicAdd(Km + Ibd, iabcd * __ldg(Pm + Iac));
            atomicAdd(Km + Ibc, iabcd * __ldg(Pm + Iad));
            atomicAdd(Km + Iad, iabcd * __ldg(Pm + Ibc));
            atomicAdd(Km + Iac, iabcd * __ldg(Pm + Ibd));
         }
      }
      __syncwarp();
   }
}

static __device__ __forceinline__ void load_plan(const ClassPlan *src_plan, double *smem) {
   const int nwords = (int)(sizeof(ClassPlan) / 4);
   const int *src = reinterpret_cast<const int *>(src_plan);
   int *dst = reinterpret_cast<int *>(smem);
   for (int w = threadIdx.x; w < nwords; w += blockDim.x) dst[w] = src[w];
}

// one warp per contraction row; the kernel waits on chains of dependent loads, so 64 registers
// (32 warps per SM, a few spills) beat 80 (24 warps)
__global__ void __launch_bounds__(256, 4) k_group(DevCtx ctx, BatchArgs bt, int warp_doubles, int use_global) {
   extern __shared__ __align__(16) double smem[];
   const ClassPlan *pl = reinterpret_cast<const ClassPlan *>(smem);
   load_plan(bt.plan, smem);
   __syncthreads();
   const int plan_doubles = (int)((sizeof(ClassPlan) + 15) / 16) * 2;
   const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarp = blockDim.x / 32;
   const int gwarp = blockIdx.x * nwarp + warp;
   // shared memory: plan | nwarp coefficient buffers | nwarp workspaces (unless in global memory)
   double *kpw = smem + plan_doubles + warp * kGroupKpDoubles;
   double *wbase = use_global ? (bt.gscratch + (size_t)gwarp * warp_doubles)
                              : (smem + plan_doubles + nwarp * kGroupKpDoubles + (size_t)warp * warp_doubles);
   const int Hws = max(pl->H, 2 * pl->Nc);
   const uint2 *hrec = ctx.gprog + ctx.gprog[bt.cls].x;
   ShellShared *cache = reinterpret_cast<ShellShared *>(kpw + 32);
   if (lane == 0) cache->key = ~0u;
   __syncwarp();
   // kGroupRowsPerWarp consecutive rows at a time, so that the rows of one set quartet that follow
   // each other on this warp reuse its group record and shell 0's shared data
   uint32_t gi = 0, gend = 0;
   GroupRec G = {};
   for (uint32_t q0 = gwarp * kGroupRowsPerWarp; q0 < bt.nqrtt; q0 += gridDim.x * nwarp * kGroupRowsPerWarp) {
      const uint32_t q1 = min(q0 + kGroupRowsPerWarp, bt.nqrtt);
      for (uint32_t q = q0; q < q1; q++) {
         if (q >= gend || q < G.qrtt_off) {
            gi = row_group_one(bt, q, lane);
            G = bt.groups[gi];
            gend = G.qrtt_off + (uint32_t)G.nl[0] * G.nl[1] * G.nl[2] * G.nl[3];
         }
         if (bt.gflags && !__ldg(bt.gflags + gi)) continue;   // screened on an incremental replay
         group_body(ctx, bt, pl, G, q, wbase, wbase + Hws, lane, hrec, kpw, cache, gi);
      }
   }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int h_ncart(int l) { return (l + 1) * (l + 2) / 2; }
static int h_cidx(int x, int y, int z) { int a = y + z; return a * (a + 1) / 2 + z; }

// Cartesian index tables for l < 8: exponents, the first axis with a nonzero exponent, and the
// index of the function one lower / one higher on each axis (-1 where that does not exist).
struct CartTables {
   int8_t exp_[8][36][3], dir[8][36], dec[8][36][3], inc[8][36][3];
};

static void make_cart_tables(CartTables &t) {
   std::memset(&t, 0, sizeof(t));
   for (int l = 0; l < 8; l++) for (int i = 0; i < 36; i++) for (int q = 0; q < 3; q++) { t.dec[l][i][q] = -1; t.inc[l][i][q] = -1; }
   for (int l = 0; l < 8; l++) {
      for (int i = 0; i < h_ncart(l); i++) {
         int a = 0; while ((a + 1) * (a + 2) / 2 <= i) a++;
         int e[3]; e[0] = l - a; e[2] = i - a * (a + 1) / 2; e[1] = a - e[2];
         for (int q = 0; q < 3; q++) t.exp_[l][i][q] = (int8_t)e[q];
         t.dir[l][i] = (int8_t)(e[0] ? 0 : (e[1] ? 1 : 2));
         for (int q = 0; q < 3; q++) {
            int f[3] = {e[0], e[1], e[2]};
            if (f[q] > 0) { f[q]--; t.dec[l][i][q] = (int8_t)h_cidx(f[0], f[1], f[2]); }
            int g[3] = {e[0], e[1], e[2]};
            g[q]++;
            if (l + 1 < 8) t.inc[l][i][q] = (int8_t)h_cidx(g[0], g[1], g[2]);
         }
      }
   }
}

// The HRR instructions of all 256 classes (layout in kernels.h). Element e of a ket step (c, d)
// is (ie, k, l) = (e / (nc nd), e / nd % nc, e % nd) and reads (ie, k + 1_t, l - 1_t) and
// (ie, k, l - 1_t); element e of a bra step (a, b) is (i, j, q) and reads (i + 1_t, j - 1_t, q)
// and (i, j - 1_t, q), t the first axis on which l (or j) has a nonzero exponent (reference
// src/compute_HRR.cpp:7-99). The steps' outputs are laid out back to back from S, so element x
// of the workspace is instruction x - S.
void build_group_prog(std::vector<uint2> &out) {
   CartTables t;
   make_cart_tables(t);
   out.assign(256, make_uint2(0u, 0u));
   for (int c = 0; c < 256; c++) {
      ClassPlan p;
      out[c].x = (uint32_t)out.size();
      if (!build_class_plan(c >> 6, (c >> 4) & 3, (c >> 2) & 3, c & 3, p)) continue;
      int x = p.S;
      for (int o = 0; o < p.nhop; o++) {
         const HOp &h = p.hop[o];
         if (h.out != x) { out.clear(); return; }   // steps not back to back: no program
         if (h.type == 0) {
            const int cc = h.x, d = h.y, nc = h_ncart(cc), nd = h_ncart(d), ncp = h_ncart(cc + 1), ndm = h_ncart(d - 1);
            for (int e = 0; e < h.nelem; e++) {
               const int l = e % nd, k = (e / nd) % nc, ie = e / (nd * nc);
               const int dr = t.dir[d][l], lm = t.dec[d][l][dr], kp = t.inc[cc][k][dr];
               const uint32_t in1 = (uint32_t)(h.in1 + (ie * ncp + kp) * ndm + lm);
               const uint32_t in2 = (uint32_t)(h.in2 + (ie * nc + k) * ndm + lm);
               out.push_back(make_uint2(in1 | ((uint32_t)dr << 30), in2));
            }
         } else {
            const int a = h.x, b = h.y, nb = h_ncart(b), nbm = h_ncart(b - 1);
            const int cdn = h_ncart(p.lc) * h_ncart(p.ld);
            for (int e = 0; e < h.nelem; e++) {
               const int q = e % cdn, j = (e / cdn) % nb, i = e / (cdn * nb);
               const int dr = t.dir[b][j], jm = t.dec[b][j][dr], ip = t.inc[a][i][dr];
               const uint32_t in1 = (uint32_t)(h.in1 + (ip * nbm + jm) * cdn + q);
               const uint32_t in2 = (uint32_t)(h.in2 + (i * nbm + jm) * cdn + q);
               out.push_back(make_uint2(in1 | ((uint32_t)dr << 30), in2));
            }
         }
         x += h.nelem;
      }
   }
}

cudaError_t upload_constant_tables(const double *c2s_l0to3, const double *symm5) {
   // the spherical passes leave out the terms outside the rows' nonzero pattern (c2s_mask)
   for (int l = 0; l <= 3; l++) {
      const int nk = h_ncart(l);
      for (int m = 0; m < 2 * l + 1; m++)
         for (int k = 0; k < nk; k++)
            if (((c2s_mask(l, m) >> k & 1) != 0) != (c2s_l0to3[l * 70 + m * nk + k] != 0.0)) return cudaErrorInvalidValue;
   }
   cudaError_t err;
   if ((err = cudaMemcpyToSymbol(c_c2s, c2s_l0to3, sizeof(double) * 4 * 70)) != cudaSuccess) return err;
   return cudaMemcpyToSymbol(c_symm, symm5, sizeof(double) * 5);
}

int plan_smem_doubles() { return (int)((sizeof(ClassPlan) + 15) / 16) * 2; }

// the opt-in shared memory per block of the first device asked (the engine's GPUs are all one
// type); a function-local static, so concurrent caller threads initialise it once
static int max_dyn_smem() {
   static const int smax = [] {
      int dev = 0, v = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      return v > 0 ? v : 48 * 1024;
   }();
   return smax;
}

// shared memory of one k_prim2 team, in doubles: cp geometries and (00|00) sums, the pair queue, one
// batch's Fm, one image's factors and the VRR workspace with its zero
static size_t prim2_team_doubles(const ClassPlan &hp, int cp) {
   const size_t w = (size_t)cp * (sizeof(PrimGeo) / 8 + 1) + 64 + 32 + 32 * (size_t)(hp.L + 1) + 18 + (size_t)hp.V + 1;
   return (w + 1) & ~(size_t)1;
}

// A workspace of this many doubles is worked on by a block instead of a warp: a warp takes a level of
// it in many rounds, and too few warps fit an SM to hide them. (1/4096 sample of 64 molecules l <= 3, primitive
// kernels one after another: 39.0 ms with warps only, 38.3; with blocks from 128 doubles on 37.2, but the
// replay, whose classes overlap, takes 58.2 instead of 57.1 ms. 256 threads from 1500 doubles on: replay 57.9;
// never: 57.1, there are few primitives of that size.)
constexpr int kPrim2BlockDoubles = 1500;
constexpr int kPrim2WideDoubles = 5000;    // and by 256 threads instead of 128 from here on
int prim_team_size(const ClassPlan &hp) { return hp.V >= kPrim2WideDoubles ? 256 : (hp.V >= kPrim2BlockDoubles ? 128 : 32); }

// Primitive-kernel choice: k_prim3 (generated VRR) for the classes it covers, else k_prim2. Its
// team is a warp for small workspaces and a block for large ones, and for segments whose chunks are
// fewer than would give every SM four warps (there one image's chain of levels is the whole time: 2 molecules
// and 27 images take 1.60 ms so and 2.19 without, 24 clusters, whose classes fill the GPU beside each other,
// 4.40 and 4.29; with 128 threads instead of 256 in the larger of these, 1.62 and 4.33).
cudaError_t launch_prim(const DevCtx &ctx, const BatchArgs &bt, const ClassPlan &hp, cudaStream_t st) {
   if (bt.nprm == 0) return cudaSuccess;
   if (bt.prim_variant == 0 || bt.fp32) {
      cudaError_t err = cudaSuccess;
      if (prim3_launch(ctx, bt, st, &err)) return err;
   }
   if (bt.fp32) return cudaErrorInvalidValue;   // FP32 segments exist only for classes with k_prim3
   // a chunk is as large as gives every resident team one, within what fills a G_m batch (about four
   // pairs a primitive with images, one without) and kPrim2Chunk; where the VRR is the larger part
   // of a primitive's time the lanes of G_m matter less than a finer split, and with fewer
   // primitives than four an SM nothing but the longest team counts
   const int fill = bt.nprm < 148u * 4 ? 1 : (hp.V >= 1000 ? 2 : 4) * (ctx.Ng == 1 ? 2 : 1);
   auto chunk = [&](long teams) { return (int)std::max((long)fill, std::min((long)kPrim2Chunk, ((long)bt.nprm + teams - 1) / teams)); };
   const size_t plan_bytes = (size_t)plan_smem_doubles() * 8;
   int cp = chunk(148 * 14);
   long nchunk = ((long)bt.nprm + cp - 1) / cp;
   if (prim_team_size(hp) > 32 || (hp.V >= 128 && nchunk < 148 * 4)) {
      cp = chunk(148 * 4);
      nchunk = ((long)bt.nprm + cp - 1) / cp;
      const size_t wd = prim2_team_doubles(hp, cp), smem = plan_bytes + wd * 8;
      const unsigned blocks = (unsigned)std::min(nchunk, 148L * 64);
      if (prim_team_size(hp) == 256 || (hp.V >= 1000 && nchunk < 148)) k_prim2<256><<<blocks, 256, smem, st>>>(ctx, bt, cp, (int)wd);
      else k_prim2<128><<<blocks, 128, smem, st>>>(ctx, bt, cp, (int)wd);
      return cudaGetLastError();
   }
   const size_t wd = prim2_team_doubles(hp, cp);
   const int nwmax = std::max(1, std::min(8, (int)((112 * 1024 - plan_bytes) / (wd * 8))));   // two blocks per SM
   const int nw = (int)std::max(1L, std::min((long)nwmax, (nchunk + 147) / 148));
   const unsigned blocks = (unsigned)std::max(1L, std::min((nchunk + nw - 1) / nw, 148L * 64));
   k_prim2<32><<<blocks, nw * 32, plan_bytes + (size_t)nw * wd * 8, st>>>(ctx, bt, cp, (int)wd);
   return cudaGetLastError();
}

size_t group_warp_doubles(const ClassPlan &hp) {
   size_t d = (size_t)std::max(hp.H, 2 * hp.Nc) + hp.Nc;
   return (d + 1) & ~(size_t)1;
}

// shared memory ahead of the group kernels' workspaces: the class plan
static size_t group_hdr_bytes() { return (size_t)plan_smem_doubles() * 8; }

// warps per block of k_group with the workspaces in shared memory (0: they do not fit)
static int group_smem_warps(size_t wd) {
   const int budget = std::min(max_dyn_smem(), 200 * 1024) - (int)group_hdr_bytes();
   return std::min(8, (int)(budget / ((wd + kGroupKpDoubles) * 8)));
}

// doubles of global scratch that k_group needs, and its launch shape there (0: the workspaces fit shared memory)
size_t group_global_scratch(const ClassPlan &hp, int *grid, int *warps) {
   const size_t wd = group_warp_doubles(hp);
   if (group_smem_warps(wd) >= 1) return 0;
   *warps = 4;
   *grid = 148 * 2;
   return wd * (size_t)(*warps) * (*grid);
}

// Group-kernel choice on variant 0: k_group3 (generated HRR, one lane per row) for the classes it
// covers, k_group_mm (one block per group) for the others; on variant 1 always
// k_group (one warp per row).
cudaError_t launch_group(const DevCtx &ctx, const BatchArgs &bt, const ClassPlan &hp, cudaStream_t st) {
   if (bt.nqrtt == 0) return cudaSuccess;
   if (bt.group_variant == 0 || bt.fp32) {
      cudaError_t err = cudaSuccess;
      if (group3_launch(ctx, bt, st, &err)) return err;
   }
   if (bt.fp32) return cudaErrorInvalidValue;   // FP32 segments exist only for classes with k_group3
   if (bt.group_variant == 0) return group_mm_launch(ctx, bt, st);
   const size_t wd = group_warp_doubles(hp);
   const size_t plan_bytes = group_hdr_bytes();
   const int nw = group_smem_warps(wd);
   if (nw >= 1) {
      const size_t smem = plan_bytes + (size_t)nw * (wd + kGroupKpDoubles) * 8;
      long blocks = ((long)bt.nqrtt + (long)nw * kGroupRowsPerWarp - 1) / ((long)nw * kGroupRowsPerWarp);
      blocks = std::max(1L, std::min(blocks, 148L * 64));
      k_group<<<(unsigned)blocks, nw * 32, smem, st>>>(ctx, bt, (int)wd, 0);
   } else {
      int grid = 0, warps = 0;
      group_global_scratch(hp, &grid, &warps);
      const size_t smem = plan_bytes + (size_t)warps * kGroupKpDoubles * 8;
      k_group<<<grid, warps * 32, smem, st>>>(ctx, bt, (int)wd, 1);
   }
   return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// Incremental replays. k_group_screen, one thread per group:
//  mode 0 (after a recording): the exact largest |P| over the P elements its rows' K updates read
//    (blocks ac: nsa x nsc, ad: nsa x nsd, bc: nsb x nsc, bd: nsb x nsd, with each row's offsets,
//    leading dimensions and transposition flags), stored in pmax;
//  mode 1 (P = dP): an upper bound of max|dP| over the same elements, from the maxima of 32-element
//    tiles of |dP| (k_tile_max) over the span of offsets each block's rows cover, and the group kept
//    unless that bound is zero or its bound scaled by it / pmax is below eps. The span bound never
//    underestimates, so no group that the exact test keeps is skipped.
// ---------------------------------------------------------------------------------------
constexpr int kScreenTile = 32;

__global__ void k_tile_max(const double *__restrict__ P, size_t n, float *__restrict__ tmax) {
   const size_t ntile = (n + kScreenTile - 1) / kScreenTile;
   const int lane = threadIdx.x & 31;
   for (size_t t = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / 32; t < ntile;
        t += (size_t)gridDim.x * blockDim.x / 32) {
      const size_t i = t * kScreenTile + lane;
      double m = i < n ? fabs(__ldg(P + i)) : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) tmax[t] = (float)(m * (1.0 + 1e-6));   // rounded up: stays an upper bound
   }
}

__global__ void k_group_screen(DevCtx ctx, BatchArgs bt, float *pmax, uint8_t *flags, double eps, int mode,
                               const float *tmax) {
   const int la = bt.cls >> 6, lb = (bt.cls >> 4) & 3, lc = (bt.cls >> 2) & 3, ld = bt.cls & 3;
   const int ns[4] = {2 * la + 1, 2 * lb + 1, 2 * lc + 1, 2 * ld + 1};
   // block u of a row: rows of centre bra[u], columns of centre ket[u] (ac, ad, bc, bd)
   const int bra[4] = {0, 0, 1, 1}, ket[4] = {2, 3, 2, 3};
   const double *Pm = ctx.P[0];
   for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < bt.ngroup; g += gridDim.x * blockDim.x) {
      const GroupRec G = bt.groups[g];
      const int nrows = G.nl[0] * G.nl[1] * G.nl[2] * G.nl[3];
      double m = 0.0;
      if (mode == 0) {
         for (int r = 0; r < nrows; r++) {
            const QrttRec k = bt.qrtts[G.qrtt_off + r];
            for (int u = 0; u < 4; u++) {
               const bool T = (k.T >> u) & 1;
               for (int i = 0; i < ns[bra[u]]; i++)
                  for (int j = 0; j < ns[ket[u]]; j++) {
                     const size_t I = (size_t)k.off[u] + (T ? i * k.ld[u] + j : j * k.ld[u] + i);
                     if (I < ctx.FP_size) m = fmax(m, fabs(__ldg(Pm + I)));
                  }
            }
         }
         pmax[g] = (float)m;
         continue;
      }
      for (int u = 0; u < 4; u++) {
         size_t lo = ~(size_t)0, hi = 0;
         for (int r = 0; r < nrows; r++) {
            const QrttRec k = bt.qrtts[G.qrtt_off + r];
            const bool T = (k.T >> u) & 1;
            const int nr = ns[bra[u]], nc = ns[ket[u]];
            const size_t a = k.off[u];
            const size_t e = a + (T ? (size_t)(nr - 1) * k.ld[u] + nc : (size_t)(nc - 1) * k.ld[u] + nr);
            lo = min(lo, a);
            hi = max(hi, e);
         }
         hi = min(hi, ctx.FP_size);
         for (size_t t = lo / kScreenTile; lo < hi && t * kScreenTile < hi; t++) m = fmax(m, (double)__ldg(tmax + t));
      }
      const double b = (double)G.bound;
      const bool skip = m == 0.0 || (isfinite(b) && b * m < eps * (double)pmax[g]);
      flags[g] = skip ? 0 : 1;
   }
}

cudaError_t launch_tile_max(const double *P, size_t n, float *tmax, cudaStream_t st) {
   const size_t ntile = (n + kScreenTile - 1) / kScreenTile;
   const long blocks = std::max(1L, std::min((long)((ntile * 32 + 255) / 256), 148L * 32));
   k_tile_max<<<(unsigned)blocks, 256, 0, st>>>(P, n, tmax);
   return cudaGetLastError();
}

size_t tile_max_count(size_t n) { return (n + kScreenTile - 1) / kScreenTile; }

// ---------------------------------------------------------------------------------------
// Merging the recorded batches of one queue class into one segment (libgint_record(h, 2)): the
// parts are copied one after another, then the indices that count within a segment are shifted
// by the part's position in the merged segment, and the per-32-row group table is rebuilt.
// ---------------------------------------------------------------------------------------
__global__ void k_rebase_part(uint32_t *prm_shell, uint32_t nprm, ShellRec *shells, uint32_t nshell, GroupRec *groups,
                              uint32_t ngroup, uint32_t prm_base, uint32_t shell_base, uint32_t group_base,
                              uint32_t qrtt_base) {
   const uint32_t n = max(nprm, max(nshell, ngroup));
   for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      if (i < nprm) prm_shell[i] += shell_base;
      if (i < nshell) { shells[i].prm_off += prm_base; shells[i].group += group_base; }
      if (i < ngroup) { groups[i].shell_off += shell_base; groups[i].qrtt_off += qrtt_base; }
   }
}

__global__ void k_row_groups(const GroupRec *groups, uint32_t ngroup, uint32_t *rowgrp) {
   for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroup; g += gridDim.x * blockDim.x) {
      const GroupRec G = groups[g];
      const uint32_t end = G.qrtt_off + (uint32_t)G.nl[0] * G.nl[1] * G.nl[2] * G.nl[3];
      for (uint32_t k = (G.qrtt_off + 31) / 32; 32 * k < end; k++) rowgrp[k] = g;
   }
}

cudaError_t launch_rebase_part(uint32_t *prm_shell, uint32_t nprm, ShellRec *shells, uint32_t nshell, GroupRec *groups,
                               uint32_t ngroup, uint32_t prm_base, uint32_t shell_base, uint32_t group_base,
                               uint32_t qrtt_base, cudaStream_t st) {
   const uint32_t n = std::max(nprm, std::max(nshell, ngroup));
   if (n == 0) return cudaSuccess;
   const long blocks = std::max(1L, std::min((long)((n + 255) / 256), 148L * 16));
   k_rebase_part<<<(unsigned)blocks, 256, 0, st>>>(prm_shell, nprm, shells, nshell, groups, ngroup, prm_base,
                                                   shell_base, group_base, qrtt_base);
   return cudaGetLastError();
}

cudaError_t launch_row_groups(const GroupRec *groups, uint32_t ngroup, uint32_t *rowgrp, cudaStream_t st) {
   if (ngroup == 0) return cudaSuccess;
   const long blocks = std::max(1L, std::min((long)((ngroup + 255) / 256), 148L * 16));
   k_row_groups<<<(unsigned)blocks, 256, 0, st>>>(groups, ngroup, rowgrp);
   return cudaGetLastError();
}

cudaError_t launch_group_screen(const DevCtx &ctx, const BatchArgs &bt, float *pmax, uint8_t *flags, double eps,
                                int mode, const float *tmax, cudaStream_t st) {
   if (bt.ngroup == 0) return cudaSuccess;
   const int threads = 128;
   const long blocks = std::max(1L, std::min(((long)bt.ngroup + threads - 1) / threads, 148L * 16));
   k_group_screen<<<(unsigned)blocks, threads, 0, st>>>(ctx, bt, pmax, flags, eps, mode, tmax);
   return cudaGetLastError();
}

// Dependent FMA chains, 8 independent chains per thread: measures the FP64 FMA pipe rate.
__global__ void k_fp64_fma(double *out, int iters, double a, double b) {
   double x[8];
#pragma unroll
   for (int i = 0; i < 8; i++) x[i] = threadIdx.x * 1e-3 + i;
   for (int it = 0; it < iters; it++) {
#pragma unroll
      for (int i = 0; i < 8; i++) x[i] = fma(x[i], a, b);
   }
   double s = 0;
#pragma unroll
   for (int i = 0; i < 8; i++) s += x[i];
   if (s == 12345.678) out[0] = s;   // keeps the chains alive
}

double measure_fp64_peak_tflops() {
   int dev = 0, sms = 0;
   cudaGetDevice(&dev);
   cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
   double *d = nullptr;
   if (cudaMalloc(&d, 8) != cudaSuccess) return 0.0;
   const int iters = 4096, threads = 512, blocks = sms * 8;
   cudaEvent_t e0, e1;
   cudaEventCreate(&e0); cudaEventCreate(&e1);
   k_fp64_fma<<<blocks, threads>>>(d, iters, 0.999999, 1e-7);   // warm-up
   float best = 1e30f;
   for (int rep = 0; rep < 5; rep++) {
      cudaEventRecord(e0);
      k_fp64_fma<<<blocks, threads>>>(d, iters, 0.999999, 1e-7);
      cudaEventRecord(e1);
      cudaEventSynchronize(e1);
      float ms = 0; cudaEventElapsedTime(&ms, e0, e1);
      best = std::min(best, ms);
   }
   cudaEventDestroy(e0); cudaEventDestroy(e1);
   cudaFree(d);
   const double flops = 2.0 * 8.0 * iters * (double)threads * blocks;
   return flops / (best * 1e-3) / 1e12;
}

// The per-device copies of the HRR instructions (build_group_prog), made once per device by
// preload_kernels and kept until the process exits.
static const uint2 *g_group_prog[kMaxDevices] = {nullptr};

static cudaError_t group_prog_load() {
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
   if (g_group_prog[dev]) return cudaSuccess;
   std::vector<uint2> prog;
   build_group_prog(prog);
   if (prog.empty()) return cudaErrorInvalidValue;
   void *p = nullptr;
   if ((e = cudaMalloc(&p, prog.size() * sizeof(uint2))) != cudaSuccess) return e;
   if ((e = cudaMemcpy(p, prog.data(), prog.size() * sizeof(uint2), cudaMemcpyHostToDevice)) != cudaSuccess) {
      cudaFree(p);
      return e;
   }
   g_group_prog[dev] = (const uint2 *)p;
   return cudaSuccess;
}

const uint2 *group_prog(int device) {
   return (device >= 0 && device < kMaxDevices) ? g_group_prog[device] : nullptr;
}

// Loads every kernel of the engine on the current device and lets each take up to the device's
// opt-in shared memory per block. The shared-memory limit is a process-wide attribute of a
// kernel: set per launch (with the launch's own size), one caller thread could lower it between
// another thread's setting and launch, which failed that launch ("invalid argument"). It is
// therefore raised once, here, before any handle launches; launches pass only their own size.
cudaError_t preload_kernels(const double *c2s_l0to3) {
   cudaError_t e;
   const int smax = max_dyn_smem();
   const void *fns[] = {(const void *)k_prim2<32>, (const void *)k_prim2<128>, (const void *)k_prim2<256>,
                        (const void *)k_group};
   for (const void *f : fns)
      if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smax)) != cudaSuccess) return e;
   cudaFuncAttributes a;
   if ((e = cudaFuncGetAttributes(&a, (const void *)k_fp64_fma)) != cudaSuccess) return e;
   if ((e = cudaFuncGetAttributes(&a, (const void *)k_rebase_part)) != cudaSuccess) return e;
   if ((e = cudaFuncGetAttributes(&a, (const void *)k_row_groups)) != cudaSuccess) return e;
   if ((e = prim3_preload(smax)) != cudaSuccess) return e;
   if ((e = group3_preload()) != cudaSuccess) return e;
   if ((e = group_mm_preload(smax, c2s_l0to3)) != cudaSuccess) return e;
   return group_prog_load();
}

// ---------------------------------------------------------------------------------------
// Fixed device scratch for libgint_replay_noalloc. Callers that cannot allocate device
// memory at K-build time (a framework that owns every device byte through its own pool, or
// code that must not trigger the implicit synchronisation of cudaMalloc/cudaFree) use this
// array instead of the handle's allocated AC/HRR buffers. It is a file-scope device array of
// kNoAllocScratchDoubles doubles (64 MiB) that every GPU which loads the library holds until
// the process exits. Host code cannot use the name g_noalloc_scratch as a device address; the
// address is obtained once per device with cudaGetSymbolAddress, with that device current.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

cudaError_t noalloc_scratch(double **ptr) {
   static std::mutex mu;
   static double *addr[kMaxDevices] = {nullptr};
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
   std::lock_guard<std::mutex> lock(mu);
   if (!addr[dev]) {
      double *p = nullptr;
      e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
      if (e != cudaSuccess) return e;
      addr[dev] = p;
   }
   *ptr = addr[dev];
   return cudaSuccess;
}

}  // namespace gint
