// Walker step for couplings of any range (sm_100a): 2D lattices on a snake path and other
// long-range Heisenberg models, with the coupling order of MPSQMC2.cpp:286-299 (by first site,
// then by second site).
//
// One CTA per walker, as in walker_step_kernel.  The centre of the walker moves left to right;
// while it sits on site i every coupling (i, j) is processed:
//   1. right environment R[j+1] = <Psi_T|phi> over sites j+1..L-1, recomputed from the first
//      still-valid one when an earlier coupling changed a site beyond j;
//   2. four left branches P[s,t] = B_i[s]^T L C[t] on the centre, carried through the middle
//      sites i+1..j-1 by ordinary transfer steps, four right branches at j and 16 closures give
//      C_kl = <Psi_T|(sqrt(s_k)U_k)_i (sqrt(s_l)V_l)_j|phi> (MPSQMC2.cpp:540-549); for
//      nearest-neighbour couplings the right branches come from the right-environment sweep, so
//      the closures are dot products only;
//   3. PDF, weight, CDF sample (551-588), O1 on the centre and O2 on site j (MPSstate.cpp:575-633).
// Then one Householder QR moves the centre to i+1, and the final site i enters the left
// environments: the trial overlap and the energy channels of the compact MPO of
// H = sum_c J_c S_i.S_j - h sum_k S^z_k (one "done" channel plus Sx, iSy, Sz per site that still
// has a partner to the right).
//
// Normalisation is deferred to the end of the step.  Every quantity the reference derives from
// the normalised walker is a ratio in which the norm cancels: PDF[x] = max(0, sum C x x) 4/(ov G)
// with C and ov of the same state, and the new overlap <Psi_T|B(x)phi> = 4 sum_kl C_kl x_k x_l.
// So the walk carries the unnormalised overlap and normalises once, when the centre reaches
// site L-1 and the norm is that of the centre.  The reference's per-coupling setOverlap
// (MPSQMC2.cpp:592) rescales by a positive number and never flips a sign here: the sampled x
// has sum C x x > 0, so the overlap stays positive.
//
// QR-free variant (p.nloff >= 0): no site is orthonormalised during the sweep.  The centre is
// stored as it is once its couplings are done, rescaled so that its squared Frobenius norm is
// its right bond dimension (that of an isometry: a per-site scale factor, carried into the FP64
// overlap), and a left norm environment Nl = sum_s A[s]^T Nl A[s] of the stored sites gives the
// norm at site L-1.  Every quantity above is gauge invariant, so the walk is the same; the host
// restores the left-canonical form (Walker::setOverlap's LeftNormalize, set_overlap_kernel) every
// few steps, which bounds the growth of the bond gauges' condition numbers.
//
// Work-buffer precision T: double (FP64 DMMA, the parity mode) or float (the mixed-precision
// sweep: site tensors, environments and branches in FP32, products on the TF32 tensor cores with
// FP32 accumulation, NP = 1 or 3 passes; the closures, PDF, sampling, weights, overlaps, norms and
// energies in FP64; walkers stay FP64 in HBM).  The mixed sweep is always QR-free.
#pragma once

#include <cfloat>
#include <type_traits>

#include "proposal.cuh"
#include "walker_kernels.cuh"

namespace mq {

template <typename T>
__device__ __forceinline__ const T *trial_of(const Dev &p) {
  if constexpr (std::is_same<T, double>::value) return p.trial;
  else return p.trial32;
}

// R[k] = sum_s B_k[s] R[k+1] A_k[s]^T from the walker's site k as stored in global memory.
// With ZB (nearest-neighbour couplings) also the right branches of site k,
// Z[s' + 2 t'] = B_k[s'] R[k+1] A_k[t']^T (a_k x b_k, ld a_k, block stride a_k * (the slot
// layout's b_k)), and R[k] = Z[0] + Z[3]: the coupling (k-1, k) then closes its left branches
// against Z[k] without products of its own (closures).  Uses Nxt and Xb.  Ends with a barrier.
template <typename T, int NP = 0, bool ZB = false>
static __device__ __forceinline__ void right_env_step(const Dev &p, SmemT<T> &s, int k) {
  const int d = kMaxD;
  {
    const int bl = s.bW[k], br = s.bW[k + 1];
    const double *W = s.W;
    load_site(s.Nxt, p.pb, s.sbC, W + s.woff[k], bl, br);
    if (k > 1) prefetch_l2(W + s.woff[k - 1], (long)s.bW[k - 1] * bl * kMaxD);  // the next site of the sweep
    __syncthreads();
    const int ar = s.aT[k + 1];
    gemm_g<NP>(ar, bl, br, cols(s.scr + s.roff[k + 1], ar), 1, cols(s.Nxt, p.pb, s.sbC), d, 1, false, s.Xb, p.pa, 0,
               s.sbX);
    __syncthreads();
  }
  const int al = s.aT[k], ar = s.aT[k + 1], bl = s.bW[k];
  const T *Bk = trial_of<T>(p) + s.toff[k];
  if constexpr (ZB) {
    {
      const long zb = (long)al * s.bS[k];
      gemm_g<NP>(al, bl, ar, cols(Bk, al, (long)al * ar), d, rows(s.Xb, p.pa, s.sbX), d, 1, false, s.scr + s.zoff[k], al,
                 zb, d * zb);
    }
    __syncthreads();
    const long zb = (long)al * s.bS[k];
    T *Rk = s.scr + s.roff[k];
    const T *Z = s.scr + s.zoff[k];
    for_block_ahead(
        al, bl, [&](int r, int c) { return Z[r + (long)al * c] + Z[3 * zb + r + (long)al * c]; },
        [&](int r, int c, T v) { Rk[r + (long)al * c] = v; });
  } else {
    gemm_g<NP>(al, bl, ar, cols(Bk, al, 0, (long)al * ar), 1, rows(s.Xb, p.pa, 0, s.sbX), 1, d, false,
               s.scr + s.roff[k], al);
  }
  __syncthreads();
}

// E_q <- sum_s F[s]^T E_q T[s] in place for n matrices E_q = E + q*ge (al x bl -> ar x br, leading
// dimension lde).  F: left factor (al x ar; K blocks s); T[s]: bl x br with column stride cs and
// sigma stride ss.  As many matrices at a time as Xb has room for.  Ends with a barrier.
template <typename T, int NP = 0>
static __device__ __forceinline__ void transfer_in_place(const Dev &p, SmemT<T> &s, const MatK<T, true> &F, int al, int ar, int bl,
                                         int br, const T *Tm, int cs, int ss, T *E, int lde, int n = 1, long ge = 0) {
  const int d = kMaxD, step = min(n, s.nx / d);
  for (int q = 0; q < n; q += step) {
    const int m = min(step, n - q);
    T *Eq = E + q * ge;
    gemm_g<NP>(al, br, bl, cols(Eq, lde, ge), m, rows(Tm, cs, ss), d, 1, false, s.Xb, p.pa, d * s.sbX, s.sbX);
    __syncthreads();
    gemm_g<NP>(ar, br, al, F, 1, rows(s.Xb, p.pa, d * s.sbX, s.sbX), m, d, false, Eq, lde, 0, ge);
    __syncthreads();
  }
}

// P[s + 2 t] = B[s]^T Lenv T[t] (ar x br) in Pb, T[t]: bl x br.  Ends with a barrier.
template <typename T, int NP = 0>
static __device__ __forceinline__ void left_branches(const Dev &p, SmemT<T> &s, const T *B, int al, int ar, int bl, int br, const T *Tm,
                                     int cs, int ss) {
  const int d = kMaxD;
  gemm_g<NP>(al, br, bl, cols(s.Lenv, p.pa), 1, rows(Tm, cs, ss), d, 1, false, s.Xb, p.pa, 0, s.sbX);
  __syncthreads();
  gemm_g<NP>(ar, br, al, rows(B, al, (long)al * ar), d, rows(s.Xb, p.pa, s.sbX), d, 1, false, s.Pb, p.pa, s.sbX,
             d * s.sbX);
  __syncthreads();
}

// The branches of the centre after the site operator O acted on it and it was scaled by inv:
// P is linear in the centre's sigma blocks, so P'[s, t] = inv sum_t' O(t, t') P[s, t'].  No barrier.
template <typename T>
static __device__ __noinline__ void mix_branches(const Dev &p, SmemT<T> &s, int ar, int br, const double *O, double inv) {
  const T o0 = T(inv * O[0]), o1 = T(inv * O[1]), o2 = T(inv * O[2]), o3 = T(inv * O[3]);
  T *P = s.Pb;
  const int pa = p.pa, sb = s.sbX;
  for_block_ahead<2>(
      ar, br,
      [&](int r, int c) {
        const T *q = P + r + pa * c;
        return Vals<T, kN2>{{q[0], q[sb], q[2 * sb], q[3 * sb]}};
      },
      [&](int r, int c, const Vals<T, kN2> &v) {
        T *q = P + r + pa * c;
#pragma unroll
        for (int sg = 0; sg < kMaxD; ++sg) {
          q[sg * sb] = o0 * v.x[sg] + o2 * v.x[sg + kMaxD];
          q[(sg + kMaxD) * sb] = o1 * v.x[sg] + o3 * v.x[sg + kMaxD];
        }
      });
}

// From the branches P of site k: Lenv' = sum_s P[s,s], the channel site k opens (its slot is none that
// closes on k) and the field's part of done'; and the lists of the site's channels.  No barrier.
template <typename T>
static __device__ __noinline__ void env_from_branches(const Dev &p, SmemT<T> &s, int k) {
  const int d = kMaxD, lda = p.maxA, ar = s.aT[k + 1], br = s.bW[k + 1];
  const long fm = (long)p.maxA * p.maxB;
  const bool init = k == 0 || p.h != 0.0;  // done' starts from the field's part
  if (threadIdx.x < 32) {  // the site's channels, in order
    const int lane = threadIdx.x, e0 = s.ech_off[k], e1 = s.ech_off[k + 1];
    int nclose = 0, ncont = 0;
    for (int base = e0; base < e1; base += 32) {
      const int e = base + lane;
      const double J = e < e1 ? p.ech_J[e] : 0.0;
      const int slot = e < e1 ? p.ech_slot[e] : 0, cont = e < e1 ? p.ech_cont[e] : 0;
      const unsigned mj = __ballot_sync(0xffffffffu, T(J) != T(0)), mc = __ballot_sync(0xffffffffu, cont != 0);
      const unsigned below = (1u << lane) - 1;
      if (mj >> lane & 1u) {
        s.closeJ[nclose + __popc(mj & below)] = J;
        s.closeS[nclose + __popc(mj & below)] = slot;
      }
      if (mc >> lane & 1u) s.contS[ncont + __popc(mc & below)] = slot;
      nclose += __popc(mj);
      ncont += __popc(mc);
    }
    if (lane == 0) {
      s.nlist[0] = nclose;
      s.nlist[1] = ncont;
    }
  }
  {
    const int op = s.eopen[k], pa = p.pa, sb = s.sbX;
    T *Fo = (op >= 0) ? s.Fch + 3L * op * fm : nullptr, *Fdn = s.Fdn, *Lenv = s.Lenv;
    const T *Pb = s.Pb;
    const T h = T(-p.h);
    T ox[kN2], oy[kN2], oz[kN2];
#pragma unroll
    for (int e = 0; e < kN2; ++e) {
      ox[e] = T(p.opSx[e]);
      oy[e] = T(p.opISy[e]);
      oz[e] = T(p.opSz[e]);
    }
    for_block_ahead<2>(
        ar, br,
        [&](int r, int c) {
          const T *q = Pb + r + pa * c;
          return Vals<T, kN2>{{q[0], q[sb], q[2 * sb], q[3 * sb]}};
        },
        [&](int r, int c, const Vals<T, kN2> &v) {
          T l = T(0), fx = T(0), fy = T(0), fz = T(0);
#pragma unroll
          for (int e = 0; e < kN2; ++e) {
            if ((e % d) == (e / d)) l += v.x[e];
            fx += ox[e] * v.x[e];
            fy += oy[e] * v.x[e];
            fz += oz[e] * v.x[e];
          }
          Lenv[r + pa * c] = l;
          if (Fo) {
            Fo[r + lda * c] = fx;
            Fo[fm + r + lda * c] = fy;
            Fo[2 * fm + r + lda * c] = fz;
          }
          if (init) Fdn[r + lda * c] = h * fz;
        });
  }
}

// G_st = delta_st Fd + sum_{i closing on k} J_ik (Sx F_i,x - iSy F_i,iy + Sz F_i,z)(s,t): G_0t in Xb[t],
// G_1t in Pb[t] (the branches are no longer needed).  No barrier.
template <typename T>
static __device__ __noinline__ void env_build(const Dev &p, SmemT<T> &s, int k) {
  const int d = kMaxD, lda = p.maxA, al = s.aT[k], bl = s.bW[k];
  const long fm = (long)p.maxA * p.maxB;
  const T *Fd = s.Fd, *Fch = s.Fch;
  T *X = s.Xb, *Y = s.Pb;
  const int pa = p.pa, sb = s.sbX, n = s.nlist[0];
  T ox[kN2], oy[kN2], oz[kN2];
#pragma unroll
  for (int e = 0; e < kN2; ++e) {
    ox[e] = T(p.opSx[e]);
    oy[e] = T(p.opISy[e]);
    oz[e] = T(p.opSz[e]);
  }
  // Four columns at a time, the channels in the outer loop: a channel's twelve reads are in flight together.
  // Element by element each read waited for the one before, 24,000 cycles at a site of the L = 64
  // chain, an eighth of its FP64 step (1,024 walkers: 24.9 ms, now 23.8 ms; 8x8 lattice unchanged).
  const int sh = al >= 32 ? 5 : 32 - __clz(al - 1), run = 1 << sh, step = blockDim.x >> sh;
  for (int r = threadIdx.x & (run - 1); r < al; r += run)
    for (int c0 = threadIdx.x >> sh; c0 < bl; c0 += 4 * step) {
      T v[4][kN2];
      int at[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        at[u] = r + lda * min(c0 + u * step, bl - 1);
        v[u][0] = Fd[at[u]];
        v[u][1] = v[u][2] = v[u][3] = T(0);
      }
      for (int e = 0; e < n; ++e) {
        const T J = T(s.closeJ[e]);
        const T *F = Fch + 3L * s.closeS[e] * fm;
        T f[4][3];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int q = 0; q < 3; ++q) f[u][q] = F[q * fm + at[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int q = 0; q < 3; ++q) v[u][q + 1] += J * f[u][q];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = c0 + u * step;
        if (c >= bl) break;
#pragma unroll
        for (int o = 0; o < kN2; ++o) {
          const int sg = o % d, tau = o / d;
          (sg == 0 ? X : Y)[tau * sb + r + pa * c] =
              ((sg == tau) ? v[u][0] : T(0)) + ox[o] * v[u][1] - oy[o] * v[u][2] + oz[o] * v[u][3];
        }
      }
    }
}

// Left environments through the final tensor Tm of site k (Tm[s] bl x br, column stride cs,
// sigma stride ss): trial overlap Lenv, "done" channel s.Fd -> s.Fdn, open channels in s.Fch
// (slot q, operator a at Fch + (3q + a) * maxA * maxB, leading dimension maxA).
// Order: branches P; from them Lenv', the channel site k opens (its slot is none that closes on k)
// and the field's part of done'; the channels that close on k, in done'; channels that stay open.
// have_P: the branches P of Tm are already in Pb (the caller derived them), skip their products.
template <typename T, int NP = 0>
static __device__ __forceinline__ void env_update_general(const Dev &p, SmemT<T> &s, int k, const T *Tm, int cs,
                                                          int ss, bool have_P = false) {
  const int d = kMaxD, lda = p.maxA;
  const long fm = (long)p.maxA * p.maxB;
  const int al = s.aT[k], ar = s.aT[k + 1], bl = s.bW[k], br = s.bW[k + 1];
  const T *B = trial_of<T>(p) + s.toff[k];
  if (!have_P) left_branches<T, NP>(p, s, B, al, ar, bl, br, Tm, cs, ss);
  env_from_branches(p, s, k);
  __syncthreads();
  if (k > 0) {
    // done' += sum_s B[s]^T (sum_t G_st Tm[t]), sum_t G_st Tm[t] in Pb[2 + s]
    const bool init = p.h != 0.0;
    env_build(p, s, k);
    __syncthreads();
    gemm_g<NP>(al, br, bl, cols(s.Xb, p.pa, s.Pb - s.Xb, s.sbX), d, rows(Tm, cs, 0, ss), 1, d, false, s.Pb + d * s.sbX, p.pa,
               s.sbX, 0);
    __syncthreads();
    gemm_g<NP>(ar, br, al, rows(B, al, 0, (long)al * ar), 1, rows(s.Pb + d * s.sbX, p.pa, 0, s.sbX), 1, d, init, s.Fdn,
               lda);
    __syncthreads();
  }
  // channels that stay open: identity on site k
  const int ncont = s.nlist[1];
  for (int e = 0; e < ncont; ++e)
    transfer_in_place<T, NP>(p, s, rows(B, al, 0, (long)al * ar), al, ar, bl, br, Tm, cs, ss,
                             s.Fch + 3L * s.contS[e] * fm, lda, 3, fm);
}

// Closures of the four left branches in Pb (cut j, a_j x b_j) with the right branches Z of site
// j (right_env_step): M[p + 4q] = <P_p, Z[q]> = <P_p, B_j[s'] R[j+1] A_j[t']^T>, q = s' + 2t'.
// Sixteen dot products in one pass, reduced in FP64.  Ends with a barrier.
template <typename T, int NP = 0>
static __device__ __noinline__ void closures_z(const Dev &p, SmemT<T> &s, int j, const T *Z) {
  const int aj = s.aT[j], bj = s.bW[j];
  const long zb = (long)aj * s.bS[j];
  double v[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = 0.0;
  {
    const T *P = s.Pb;
    const int pa = p.pa, sb = s.sbX;
    for_block_ahead<2>(
        aj, bj,
        [&](int m, int n) {
          const T *q = P + m + pa * n, *z = Z + m + (long)aj * n;
          return Vals<T, 2 * kN2>{{q[0], q[sb], q[2 * sb], q[3 * sb], z[0], z[zb], z[2 * zb], z[3 * zb]}};
        },
        [&](int, int, const Vals<T, 2 * kN2> &x) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k + 4 * q] += (double)x.x[k] * (double)x.x[4 + q];
        });
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < 16; ++q)
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < 16; ++q) s.red[q * nw + warp] = v[q];
  add_warps(s.red, s.M);
}

// The same closures for couplings of any range: the right branches of site j (walker site in
// Nxt, R[j+1] at Rn) formed and dotted with P in one pass of products.
template <typename T, int NP = 0>
static __device__ __forceinline__ void closures_products(const Dev &p, SmemT<T> &s, int j, const T *Rn) {
  const int d = kMaxD;
  const int aj = s.aT[j], a2 = s.aT[j + 1], bj = s.bW[j], b2 = s.bW[j + 1];
  const T *Bj = trial_of<T>(p) + s.toff[j];
  gemm_g<NP>(a2, bj, b2, cols(Rn, a2), 1, cols(s.Nxt, p.pb, s.sbC), d, 1, false, s.Xb, p.pa, 0, s.sbX);
  __syncthreads();
  // M[k + 4 (s' + 2 t')] = <P_k, B_j[s'] Y[t']>, the products formed and dotted in one pass
  cta_closure16<NP>(aj, bj, a2, Bj, aj, aj * a2, s.Xb, p.pa, s.sbX, s.Pb, p.pa, s.sbX, s.red, s.M);
}

// The 16 closures of coupling (i, j), left branches in Pb: against the stored right branches of
// site j (ZB) or formed here (site j from W, R[j+1] from the scratch).  Uses Nxt and Xb.
template <typename T, int NP = 0, bool ZB = false>
static __device__ __forceinline__ void closures(const Dev &p, SmemT<T> &s, int j) {
  if constexpr (ZB) {
    closures_z<T, NP>(p, s, j, s.scr + s.zoff[j]);
  } else {
    load_site(s.Nxt, p.pb, s.sbC, s.W + s.woff[j], s.bW[j], s.bW[j + 1]);
    __syncthreads();
    closures_products<T, NP>(p, s, j, s.scr + s.roff[j + 1]);
  }
}

// Largest v over the CTA (every thread gets it).  red: >= kWarps doubles.
__device__ __forceinline__ double cta_max(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double m = red[0];
#pragma unroll
  for (int w = 1; w < kWarps; ++w) m = fmax(m, red[w]);
  return m;
}

// C_kl = sqrt(s_k s_l) sum U_k M V_l from the closures (16 threads).  Ends with a barrier.
template <typename T>
__device__ __forceinline__ void coupling_matrix(const Dev &p, SmemT<T> &s, int jq) {
  const int tid = threadIdx.x;
  const double *U = s.tabU + 16 * jq, *Sq = s.tabSq + 4 * jq, *VT = s.tabVT + 16 * jq;
  if (tid < 16) {
    const int k = tid & 3, l = tid >> 2;
    double acc = 0.0;
    for (int qq = 0; qq < 4; ++qq) {
      double inner = 0.0;
      for (int pp = 0; pp < 4; ++pp) inner += U[pp + 4 * k] * s.M[pp + 4 * qq];
      acc += inner * VT[l + 4 * qq];
    }
    s.Cm[k + 4 * l] = Sq[k] * Sq[l] * acc;
  }
  __syncthreads();
}

// The sampled grid point's numbers for the CTA: index, uniform, weight factor, the walker's new
// (unnormalised) overlap 4 sum_kl C_kl x_k x_l and weight, and the site operators O1(s,t) = sum_k sqrt(4 s_k) x_k U_k, O2 likewise (one warp; lane q < 4
// forms O1[q], lane 4 + q O2[q]).
template <typename T>
__device__ __forceinline__ void take_point(const Dev &p, SmemT<T> &s, int jq, int count, double u, double factor) {
  const int lane = threadIdx.x & 31;
  const double *U = s.tabU + 16 * jq, *Sq = s.tabSq + 4 * jq, *VT = s.tabVT + 16 * jq;
  const double *x = s.grid + 4 * count;
  if (lane < 8) {
    const int q = lane & 3;
    double o = 0.0;
    for (int k = 0; k < 4; ++k) o += 2.0 * Sq[k] * x[k] * (lane < 4 ? U[q + 4 * k] : VT[k + 4 * q]);
    (lane < 4 ? s.O1 : s.O2)[q] = o;
  } else if (lane == 8) {
    double nm = 0.0;
    for (int l = 0; l < 4; ++l) {
      double row = 0.0;
      for (int r = 0; r < 4; ++r) row += s.Cm[l + 4 * r] * x[r];
      nm += row * x[l];
    }
    s.sc[2] = count;
    s.sc[3] = u;
    s.sc[4] = factor;
    s.sc[kScOv] = 4.0 * nm;
    s.sc[kScWt] *= factor;
  }
}

// The point where the warp's scan (sample_grid) found none (from == G) or one of probability zero (from): the
// next of nonzero probability, or the last one; and where the sum of the PDF is zero, infinite or no
// number, the point at which the serial scan's comparisons end.
static __device__ __noinline__ int rare_point(const double *pdf, int G, int per, int from, double pinv, double u) {
  auto at = [&](int g) { return pdf[32 * (g % per) + g / per]; };
  int g = from;
  if (!(pinv > 0.0 && pinv <= DBL_MAX)) {
    g = 0;
    for (double cum = at(0) * pinv; cum <= u && g < G - 1; cum += at(g) * pinv) ++g;
    return g;
  }
  while (g < G && at(g) == 0.0) ++g;
  if (g >= G)
    for (g = G - 1; g > 0 && at(g) == 0.0;) --g;
  return g;
}

// C_kl from the closures, PDF over the grid, weight update, CDF sample with the walker's uniform
// for coupling c, and the site operators O1, O2 (MPSQMC2.cpp:551-588, MPSstate.cpp:575-633).
// The CDF scan is one warp's: lane k holds the run of grid points from k*per on (stored per-major,
// so that its reads are free of conflicts), a prefix sum over the lanes places the run, and the
// first lane whose running sum passes u has the point (a serial scan by one thread took 7,000
// cycles of a coupling on average).  The sum in front of a lane and the last running sum of the lane
// before it are rounded differently; a uniform between the two goes to the next point of nonzero
// probability (behind the last sum: to the last such point), as the sampled point's sum C x x has to
// be positive.
template <typename T>
static __device__ __noinline__ void sample_grid(const Dev &p, SmemT<T> &s, int c, int jq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned full = 0xffffffffu;
  coupling_matrix(p, s, jq);
  const double fac = 4.0 / (s.sc[kScOv] * p.G);
  const int per = (p.G + 31) >> 5;
  for (int i = warp; i < per; i += nw) {
    const int g = lane * per + i;
    double v = 0.0;
    if (g < p.G) {
      const double *x = s.grid + 4 * g;
      for (int l = 0; l < 4; ++l) {
        double row = 0.0;
        for (int r = 0; r < 4; ++r) row += s.Cm[l + 4 * r] * x[r];
        v += row * x[l];
      }
    }
    s.pdf[32 * i + lane] = fmax(0.0, v) * fac;
  }
  __syncthreads();
  if (warp == 0) {
    const double u = p.uni[(long)s.w * p.nC + c];
    double run = 0.0;
    for (int i = 0; i < per; ++i) run += s.pdf[32 * i + lane];
    double cum = run;
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(full, cum, o);
      if (lane >= o) cum += y;
    }
    const double pnorm = __shfl_sync(full, cum, 31), pinv = 1.0 / pnorm;
    double at = __shfl_up_sync(full, cum, 1);
    if (lane == 0) at = 0.0;
    int hit = per;
    for (int i = 0; i < per; ++i) {
      at += s.pdf[32 * i + lane];
      if (hit == per && at * pinv > u) hit = i;
    }
    const unsigned who = __ballot_sync(full, hit < per);
    const int src = __ffs(who) - 1, h = __shfl_sync(full, hit, src & 31);
    int count = src * per + h;
    if (!who || s.pdf[32 * h + src] == 0.0) count = rare_point(s.pdf, p.G, per, who ? count : p.G, pinv, u);
    take_point(p, s, jq, count, u, pnorm);
  }
  __syncthreads();
}

// The same with the learned proposal or its training on (256 threads).  Learned proposal (p.prop_mode == 1, proposal.cuh): the point is drawn from the network's q~ on
// the support of the PDF and the weight takes P(x) / q~(x); with p.prop_collect the grid walk
// stores the features and the normalised PDF of coupling w % nC as a training pair.
template <typename T>
static __device__ void sample_learned(const Dev &p, SmemT<T> &s, int c, int jq) {
  const int tid = threadIdx.x, w = s.w;
  const double ov = s.sc[kScOv];
  coupling_matrix(p, s, jq);
  const double fac = 4.0 / (ov * p.G);
  double part = 0.0;
  for (int g = tid; g < p.G; g += kThreads) {
    const double *x = p.grid + 4 * g;
    double v = 0.0;
    for (int l = 0; l < 4; ++l)
      for (int r = 0; r < 4; ++r) v += s.Cm[l + 4 * r] * x[l] * x[r];
    v = fmax(0.0, v) * fac;
    s.pdf[g] = v;
    part += v;
  }
  const double pnorm = cta_sum(part, s.red);
  const bool learned = p.prop_mode == 1;
  const bool collect = !learned && p.prop_collect && c == w % p.nC;
  if (learned || collect) {  // the 32 features
    float *f = s.mlp;
    if (tid < 16) f[tid] = (float)(4.0 * s.Cm[tid] / ov);
    else if (tid < 32) f[tid] = (float)(4.0 * s.M[tid - 16] / ov);
    __syncthreads();
    if (collect)
      for (int e = tid; e < kMlpIn; e += kThreads) p.prop_feat[(long)w * kMlpIn + e] = f[e];
  }
  if (!learned) {
    const double pinv = 1.0 / pnorm;
    for (int g = tid; g < p.G; g += kThreads) {
      s.pdf[g] *= pinv;
      if (collect) p.prop_target[(long)w * p.G + g] = (float)s.pdf[g];
    }
    __syncthreads();
  } else {
    float *z = s.mlp + kMlpIn + 4 * kMlpHid;
    mlp_forward_cta(p.prop_w, p.G, s.mlp, s.mlp + kMlpIn, s.mlp + kMlpIn + 2 * kMlpHid, z);
    double zmax = -INFINITY;
    for (int g = tid; g < p.G; g += kThreads)
      if (s.pdf[g] > 0.0) zmax = fmax(zmax, (double)z[g]);
    zmax = cta_max(zmax, s.red);
    double se = 0.0;
    for (int g = tid; g < p.G; g += kThreads) {
      const double e = (s.pdf[g] > 0.0) ? exp((double)z[g] - zmax) : 0.0;
      s.qprop[g] = e;
      se += e;
    }
    // the defensive mixture (1 - alpha) q~ + alpha P / sum P: P / q_mix <= sum P / alpha
    const double qinv = (1.0 - p.prop_mix) / cta_sum(se, s.red), pinv = pnorm > 0.0 ? p.prop_mix / pnorm : 0.0;
    for (int g = tid; g < p.G; g += kThreads) s.qprop[g] = s.qprop[g] * qinv + s.pdf[g] * pinv;
    __syncthreads();
  }
  if (tid == 0) {
    const double u = p.uni[(long)w * p.nC + c];
    int count = 0;
    double factor = pnorm;
    if (!learned) {
      double cum = s.pdf[0];
      while ((cum <= u) && (count < p.G - 1)) {
        count += 1;
        cum += s.pdf[count];
      }
    } else {
      // first support point whose cumulative q~ exceeds u (the last one if rounding leaves u above)
      double cum = 0.0;
      int last = 0;
      for (int g = 0; g < p.G; ++g) {
        if (s.qprop[g] <= 0.0) continue;
        last = g;
        cum += s.qprop[g];
        if (cum > u) break;
      }
      count = last;
      factor = s.pdf[count] / s.qprop[count];
    }
    s.sc[6] = count;
    s.sc[7] = factor;
  }
  __syncthreads();
  if (tid < 32) take_point(p, s, jq, (int)s.sc[6], p.uni[(long)w * p.nC + c], s.sc[7]);
  __syncthreads();
}

template <typename T, bool LEARN>
__device__ __forceinline__ void sample_coupling(const Dev &p, SmemT<T> &s, int c, int jq) {
  if (LEARN && (p.prop_mode == 1 || p.prop_collect)) sample_learned(p, s, c, jq);
  else sample_grid(p, s, c, jq);
}

// Site operator O (2x2, O[s + 2t]) on a site held in smem (rows r < dl, columns < dr, sigma
// stride sb, column stride ld), in place.  No barrier.
template <typename T>
__device__ __forceinline__ void apply_site_op(T *X, int ld, int sb, int dl, int dr, const double *O) {
  const T o0 = T(O[0]), o1 = T(O[1]), o2 = T(O[2]), o3 = T(O[3]);
  for_block_ahead(
      dl, dr, [&](int r, int c) { return Vals<T, 2>{{X[r + ld * c], X[sb + r + ld * c]}}; },
      [&](int r, int c, const Vals<T, 2> &v) {
        X[r + ld * c] = o0 * v.x[0] + o2 * v.x[1];
        X[sb + r + ld * c] = o1 * v.x[0] + o3 * v.x[1];
      });
}

// The same on a site as stored in HBM (X[r + dl (c + dr sigma)], FP64), in place.  No barrier.
__device__ __forceinline__ void apply_site_op_stored(double *X, int dl, int dr, const double *O) {
  const int blk = dl * dr;
  const double o0 = O[0], o1 = O[1], o2 = O[2], o3 = O[3];
  for_block_ahead(
      dl, dr, [&](int r, int c) { return Vals<double, 2>{{X[r + dl * c], X[blk + r + dl * c]}}; },
      [&](int r, int c, const Vals<double, 2> &v) {
        X[r + dl * c] = o0 * v.x[0] + o2 * v.x[1];
        X[blk + r + dl * c] = o1 * v.x[0] + o3 * v.x[1];
      });
}

// Centre on site 0: overlap <Psi_T|phi> (the stored walker is normalised, overlap > 0), Lenv = 1.
// No barrier at the end.
template <typename T>
static __device__ __noinline__ void first_overlap(const Dev &p, SmemT<T> &s) {
  const int d = kMaxD, tid = threadIdx.x;
  const int a1 = s.aT[1], b1 = s.bW[1];
  load_site(s.Cen, p.pb, s.sbC, s.W + s.woff[0], 1, b1);
  __syncthreads();
  const T *R1 = s.scr + s.roff[1], *B0 = trial_of<T>(p) + s.toff[0];
  double part = 0.0;
  for (int q = tid; q < a1 * b1 * d; q += blockDim.x) {
    const int a = q % a1, rest = q / a1, b = rest % b1, sg = rest / b1;
    part += (double)B0[a + a1 * sg] * (double)R1[a + a1 * b] * (double)s.Cen[sg * s.sbC + p.pb * b];
  }
  const double ov = cta_sum(part, s.red);
  if (tid == 0) {
    s.sc[kScOv] = ov;
    s.Lenv[0] = T(1);
  }
}

// The centre as the final site i: rescaled to the Frobenius norm of an isometry (sqrt(br)), so that the
// tensor scales cannot drift over the steps (the overlap takes the same factor), and stored; its
// branches with it when Pb holds those of the last coupling.  No barrier at the end.
template <typename T>
static __device__ __noinline__ void rescale_centre(const Dev &p, SmemT<T> &s, int i, bool branches_kept) {
  constexpr bool kMixed = !std::is_same<T, double>::value;
  const int tid = threadIdx.x;
  const int bl = s.bW[i], br = s.bW[i + 1], sbC = s.sbC;
  double *Wi = s.W + s.woff[i];
  T *C = s.Cen;
  double part = 0.0;
  const int blk = bl * br;
  auto get = [&](int r, int cc) {
    const double *y = Wi + r + bl * cc;
    const T *x = C + r + p.pb * cc;
    return kMixed ? Vals<double, 2>{{y[0], y[blk]}} : Vals<double, 2>{{(double)x[0], (double)x[sbC]}};
  };
  for_block_ahead(bl, br, get, [&](int, int, const Vals<double, 2> &v) { part += v.x[0] * v.x[0] + v.x[1] * v.x[1]; });
  const double inv = sqrt((double)br / cta_sum(part, s.red));
  for_block_ahead(bl, br, get, [&](int r, int cc, const Vals<double, 2> &v) {
    double *y = Wi + r + bl * cc;
    T *x = C + r + p.pb * cc;
    x[0] *= T(inv);
    x[sbC] *= T(inv);
    y[0] = kMixed ? v.x[0] * inv : (double)x[0];  // the stored site
    y[blk] = kMixed ? v.x[1] * inv : (double)x[sbC];
  });
  if (tid == 0) {
    s.sc[kScOv] *= inv;
    s.sc[kScNorm] *= inv;
  }
  if (branches_kept) mix_branches(p, s, s.aT[i + 1], br, s.O1, inv);
}

// The last site i: overlap, weight and local energy out, the centre normalised and stored (its norm
// through Nl, or its own after a QR per site).
template <typename T>
static __device__ __noinline__ void finish_walker(const Dev &p, SmemT<T> &s, int i) {
  constexpr bool kMixed = !std::is_same<T, double>::value;
  const int d = kMaxD, tid = threadIdx.x;
  const int bl = s.bW[i], sbC = s.sbC;
  double *Wi = s.W + s.woff[i];
  T *C = s.Cen;
  const T *Nl = s.Nl;
  double part = 0.0;
  for (int q = tid; q < bl * d; q += blockDim.x) {  // site L-1: bl x 1 per sigma
    const T *cs = C + (q / bl) * sbC;
    const double *ws = Wi + (q / bl) * bl;  // the FP64 walker (mixed sweep)
    const double x = kMixed ? ws[q % bl] : (double)cs[q % bl];
    if (Nl == nullptr) {
      part += x * x;
    } else {  // x (Nl c)_r
      double y = 0.0;
      for (int k = 0; k < bl; ++k) y += (double)Nl[(q % bl) + p.pb * k] * (kMixed ? ws[k] : (double)cs[k]);
      part += x * y;
    }
  }
  const double nrm = sqrt(cta_sum(part, s.red));
  const double ovr = s.Lenv[0];
  const double en = s.Fdn[0];
  const double scale = (ovr < 0.0) ? -1.0 / nrm : 1.0 / nrm;
  if (kMixed) {
    for (int q = tid; q < bl * d; q += blockDim.x) Wi[q] *= scale;
  } else {
    for (int q = tid; q < bl * d; q += blockDim.x) C[(q / bl) * sbC + (q % bl)] *= T(scale);
    __syncthreads();
    store_site(Wi, C, p.pb, sbC, bl, 1);
  }
  if (tid == 0) {
    const double ovf = fabs(ovr) / nrm;
    const double ew = en / ovr, wt = s.sc[kScWt];
    p.overlap[s.slot] = ovf;
    p.weight[s.slot] = wt;
    p.energy[s.w] = ew;
    p.ov_out[s.w] = ovf;
    p.wt_out[s.w] = wt;
    if (!(isfinite(wt) && isfinite(ovf) && isfinite(ew))) atomicOr(p.err, kErrNumeric);
  }
}

// ||phi||^2 of the walker with the centre C on site i (sites > i as stored in global memory):
// N = sum_s A_k[s] N A_k[s]^T from site L-1 down to i+1 (in the norm-environment scratch), then
// sum_s tr(C[s]^T Nl C[s] N) with the left norm environment Nl of sites < i (ld pb), or the
// identity when those sites are orthonormal (Nl == nullptr).  Uses Nxt, Xb, Pb.  Only the trace
// mode calls it, to report the reference's normalised C_kl and overlaps.
template <typename T, int NP = 0>
static __device__ double norm_from_centre(const Dev &p, SmemT<T> &s, int i, const T *Nl = nullptr) {
  const double *W = s.W;
  T *scr = s.scr;
  const int L = p.L, d = kMaxD, tid = threadIdx.x;
  if (tid == 0) scr[p.nroff[L]] = T(1);
  __syncthreads();
  for (int k = L - 1; k > i; --k) {
    const int bl = s.bW[k], br = s.bW[k + 1];
    load_site(s.Nxt, p.pb, s.sbC, W + s.woff[k], bl, br);
    __syncthreads();
    const T *Nn = scr + p.nroff[k + 1];
    T *Nk = scr + p.nroff[k];
    gemm_g<NP>(br, bl, br, cols(Nn, br), 1, cols(s.Nxt, p.pb, s.sbC), d, 1, false, s.Pb, p.pa, 0, s.sbX);
    __syncthreads();
    gemm_g<NP>(bl, bl, br, cols(s.Nxt, p.pb, 0, s.sbC), 1, rows(s.Pb, p.pa, 0, s.sbX), 1, d, false, Nk, bl);
    __syncthreads();
  }
  const int bl = s.bW[i], br = s.bW[i + 1];
  const T *N1 = scr + p.nroff[i + 1];
  gemm_g<NP>(bl, br, br, cols(s.Cen, p.pb, s.sbC), d, rows(N1, br), 1, 1, false, s.Xb, p.pa, s.sbX, 0);
  __syncthreads();
  const T *Z = s.Xb;
  if (Nl != nullptr) {
    gemm_g<NP>(bl, br, bl, cols(Nl, p.pb), 1, rows(s.Xb, p.pa, s.sbX), d, 1, false, s.Pb, p.pa, 0, s.sbX);
    __syncthreads();
    Z = s.Pb;
  }
  double part = 0.0;
  for_block(bl, br, [&](int r, int cc) {
    for (int sg = 0; sg < d; ++sg)
      part += (double)s.Cen[sg * s.sbC + r + p.pb * cc] * (double)Z[sg * s.sbX + r + p.pa * cc];
  });
  return cta_sum(part, s.red);
}

#ifndef MQ_DEVICE_ONLY

// The walker step (all walkers of the population, one CTA per walker at a time).
// QM: 1 the QR-free sweep, 0 QR-free or a QR per site, chosen by p.nloff at run time.  TR: the
// per-coupling trace is compiled in (recorded when p.trace is set).  LEARN: the learned proposal
// and its training are compiled in.
template <typename T, int NP, bool ZB, int QM, bool TR, bool LEARN>
__device__ __forceinline__ void general_step(const Dev &args, double *smem_raw) {
  const Dev &p = shared_args(smem_raw);
  constexpr bool kMixed = !std::is_same<T, double>::value;
  SmemT<T> &s = *reinterpret_cast<SmemT<T> *>(smem_raw);
  carve_shared<T, QM == 1 && !kMixed>(args, smem_raw);
  const bool QF = QM == 1 || args.nloff >= 0;
  const bool traced = TR && args.trace != nullptr;
  const int L = p.L, d = kMaxD, tid = threadIdx.x;
  for (;;) {
    const int w = next_walker(s, p.ctr + kCtrStep);
    if (w >= *p.n_cur) break;
    {
      const int slot = p.slot_of[w];
      load_walker_dims(p, s, slot);
      if (tid == 0) {
        T *scr = reinterpret_cast<T *>(p.scratch) + (long)blockIdx.x * p.scr_stride;
        const long fm = (long)p.maxA * p.maxB;
        s.w = w;
        s.slot = slot;
        s.W = p.walkers + (long)slot * p.wstride;
        s.scr = scr;
        s.Fd = scr + p.choff;
        s.Fdn = s.Fd + fm;
        s.Fch = s.Fdn + fm;
        if (QM != 1 || kMixed) s.Nl = QF ? scr + p.nloff : nullptr;
      }
      if (tid == 0) {
        s.scr[s.roff[L]] = T(1);
        if (QF) s.Nl[0] = T(1);
        s.sc[kScWt] = p.weight[slot];
      }
      __syncthreads();
    }
    // right environments of the walker as stored
    for (int k = L - 1; k >= 1; --k) right_env_step<T, NP, ZB>(p, s, k);
    int rv = 1;  // R[k] is valid for k >= rv
    first_overlap(p, s);
    if (traced) {  // kScNorm: norm of the walker before the current coupling
      const double nrm = sqrt(norm_from_centre<T, NP>(p, s, 0));
      if (tid == 0) s.sc[kScNorm] = nrm;
    }
    __syncthreads();
    for (int i = 0; i < L; ++i) {
      // the walker's next site, and on chains the right branches this site's coupling closes with
      // (formed in the right-environment sweep, since evicted from L2): fetched ahead
      if (i + 1 < L) {
        const int br = s.bW[i + 1];
        prefetch_l2(s.W + s.woff[i + 1], (long)br * s.bW[i + 2] * d);
        if constexpr (ZB)
          for (int q = 0; q < kN2; ++q)
            prefetch_l2(s.scr + s.zoff[i + 1] + (long)q * s.aT[i + 1] * s.bS[i + 1], (long)s.aT[i + 1] * br);
      }
      // Pb still holds the last coupling's left branches at cut i+1 (its partner was i+1, so they
      // were not carried further, and the trace did not use Pb as scratch)
      bool branches_kept = false;
      for (int c = s.site_c0[i]; c < s.site_c0[i + 1]; ++c) {
        const int j = s.cp_j[c];
        while (rv > (ZB ? j : j + 1)) {  // R[j+1] (and the right branches of site j) up to date
          --rv;
          right_env_step<T, NP, ZB>(p, s, rv);
        }
        if constexpr (!ZB) {  // what the closures read after the middle sites: site j and R[j+1]
          if (j > i + 1) prefetch_l2(s.W + s.woff[j], (long)s.bW[j] * s.bW[j + 1] * d);
          prefetch_l2(s.scr + s.roff[j + 1], (long)s.aT[j + 1] * s.bW[j + 1]);
        }
        // left branches P[s + d t] = B_i[s]^T Lenv C[t] (a_{i+1} x b_{i+1}); after a coupling with the
        // next site they are that coupling's, mixed by its O1 (in FP64; the FP32 sweep keeps its roundings)
        if (!kMixed && branches_kept) {
          mix_branches(p, s, s.aT[i + 1], s.bW[i + 1], s.O1, 1.0);
          __syncthreads();
        } else {
          left_branches<T, NP>(p, s, trial_of<T>(p) + s.toff[i], s.aT[i], s.aT[i + 1], s.bW[i], s.bW[i + 1], s.Cen, p.pb,
                               s.sbC);
        }
        // through the middle sites
        for (int m = i + 1; m < j; ++m) {
          const int am = s.aT[m], am1 = s.aT[m + 1], bm = s.bW[m], bm1 = s.bW[m + 1];
          load_site(s.Nxt, p.pb, s.sbC, s.W + s.woff[m], bm, bm1);
          if (m + 1 < j) prefetch_l2(s.W + s.woff[m + 1], (long)bm1 * s.bW[m + 2] * d);
          __syncthreads();
          transfer_in_place<T, NP>(p, s, rows(trial_of<T>(p) + s.toff[m], am, 0, (long)am * am1), am, am1, bm, bm1, s.Nxt,
                                   p.pb, s.sbC, s.Pb, p.pa, kN2, s.sbX);
        }
        // closures with the right branches of site j, sample, site operators
        closures<T, NP, ZB>(p, s, j);
        sample_coupling<T, LEARN>(p, s, c, s.cp_q[c]);
        apply_site_op(s.Cen, p.pb, s.sbC, s.bW[i], s.bW[i + 1], s.O1);
        // O2 acts on site j as stored in HBM; in the mixed sweep the walker itself stays FP64, so
        // O1 acts on its stored site i as well (the FP32 centre only feeds the contractions)
        if constexpr (kMixed) apply_site_op_stored(s.W + s.woff[i], s.bW[i], s.bW[i + 1], s.O1);
        apply_site_op_stored(s.W + s.woff[j], s.bW[j], s.bW[j + 1], s.O2);
        __syncthreads();
        if (rv < j + 1) rv = j + 1;
        branches_kept = (j == i + 1) && !traced;
        if (traced) {
          // the reference normalises after every coupling: report C of the normalised walker
          // and the normalised overlap (the walk itself does not need the norm)
          const double nrm_after = sqrt(norm_from_centre<T, NP>(p, s, i, s.Nl));
          if (tid == 0) {
            double *t = p.trace + ((long)w * p.nC + c) * kTraceStride;
            for (int k = 0; k < 16; ++k) t[k] = s.Cm[k] / s.sc[kScNorm];
            t[16] = s.sc[4];
            t[17] = s.sc[3];
            t[18] = s.sc[2];
            t[19] = s.sc[kScWt];
            t[20] = s.sc[kScOv] / nrm_after;
            s.sc[kScNorm] = nrm_after;
          }
          __syncthreads();
        }
      }
      if (QF && i < L - 1) {
        // QR-free: the centre itself becomes the final site i, and the left norm environment takes it
        // in: Nl' = sum_s C[s]^T Nl C[s]
        rescale_centre(p, s, i, branches_kept);
        __syncthreads();
        {
          const int bl = s.bW[i], br = s.bW[i + 1];
          transfer_in_place<T, NP>(p, s, rows(s.Cen, p.pb, 0, s.sbC), bl, br, bl, br, s.Cen, p.pb, s.sbC, s.Nl, p.pb);
        }
        env_update_general<T, NP>(p, s, i, s.Cen, p.pb, s.sbC, branches_kept);
        load_site(s.Cen, p.pb, s.sbC, s.W + s.woff[i + 1], s.bW[i + 1], s.bW[i + 2]);
      } else if (i < L - 1) {
        if constexpr (std::is_same<T, double>::value && QM != 1) {
          // QR of the centre: Q is the final site i, R moves into site i+1
          const int bl = s.bW[i], br = s.bW[i + 1];
          for (int q = tid; q < bl * br; q += kThreads) {
            const int r = q % bl, cc = q / bl;
            s.QRb[(r + bl * 0) + p.pq * cc] = s.Cen[r + p.pb * cc];
            s.QRb[(r + bl * 1) + p.pq * cc] = s.Cen[s.sbC + r + p.pb * cc];
          }
          __syncthreads();
          cta_householder_qr(bl * d, br, s.QRb, p.pq, s.Rf, p.pb, s.tau);
          double *Wi = s.W + s.woff[i];
          for (int q = tid; q < bl * br * d; q += kThreads) {
            const int r = q % bl, rest = q / bl, cc = rest % br, sg = rest / br;
            Wi[q] = s.QRb[(r + bl * sg) + p.pq * cc];
          }
          const int b2 = s.bW[i + 2];
          load_site(s.Nxt, p.pb, s.sbC, s.W + s.woff[i + 1], br, b2);
          __syncthreads();
          gemm_g<NP>(br, b2, br, cols(s.Rf, p.pb), 1, rows(s.Nxt, p.pb, s.sbC), d, 1, false, s.Cen, p.pb, 0, s.sbC);
          __syncthreads();
          env_update_general<T, NP>(p, s, i, s.QRb, p.pq, bl);
        }
      } else {
        // last site: energy and overlap of the unnormalised walker, then normalise the centre
        env_update_general<T, NP>(p, s, i, s.Cen, p.pb, s.sbC);
        finish_walker(p, s, i);
      }
      if (tid == 0) {  // the "done" channel changes places
        T *f = s.Fd;
        s.Fd = s.Fdn;
        s.Fdn = f;
      }
      __syncthreads();
    }
  }
}

// The FP64 walk: QR-free, no trace, the grid proposal.  ZB: nearest-neighbour couplings, right
// branches stored per site.  128 registers a thread, so that 512 threads of several walkers share an
// SM (capi.cu, layout_free).
template <bool ZB>
__global__ void __launch_bounds__(32 * kMaxWarps, 1) walker_step_kernel_fp64(Dev p) {
  extern __shared__ double smem_raw[];
  general_step<double, 0, ZB, 1, false, false>(p, smem_raw);
}

// The FP64 walk with the QR per site, the trace or the learned proposal, as asked for at run time.
template <bool ZB>
__global__ void __launch_bounds__(kThreads, 1) walker_step_general_kernel(Dev p) {
  extern __shared__ double smem_raw[];
  general_step<double, 0, ZB, 0, true, true>(p, smem_raw);
}

// Mixed precision: FP32 work buffers, TF32 tensor cores (NP passes), always QR-free.  Half the
// matrix buffers' bytes, so two CTAs of 256 threads fit on an SM where they would be one in FP64.
template <int NP, bool ZB>
__global__ void __launch_bounds__(kThreads, 2) walker_step_mixed_kernel(Dev p) {
  extern __shared__ double smem_raw[];
  general_step<float, NP, ZB, 1, true, true>(p, smem_raw);
}

// <Psi_T|H|phi> / overlap for every walker (any coupling range), tensors as stored.
__global__ void __launch_bounds__(32 * kMaxWarps, 1) energy_general_kernel(Dev args) {
  extern __shared__ double smem_raw[];
  Smem &s = *reinterpret_cast<Smem *>(smem_raw);
  carve_shared<double, true>(args, smem_raw);
  const Dev &p = shared_args(smem_raw);
  const int L = p.L, tid = threadIdx.x;
  for (;;) {
    const int w = next_walker(s, p.ctr + kCtrEnergy);
    if (w >= *p.n_cur) break;
    const int slot = p.slot_of[w];
    load_walker_dims(p, s, slot);
    if (tid == 0) {
      s.W = p.walkers + (long)slot * p.wstride;
      s.Fd = p.scratch + (long)blockIdx.x * p.scr_stride + p.choff;
      s.Fdn = s.Fd + (long)p.maxA * p.maxB;
      s.Fch = s.Fdn + (long)p.maxA * p.maxB;
      s.Lenv[0] = 1.0;
    }
    __syncthreads();
    for (int k = 0; k < L; ++k) {
      load_site(s.Cen, p.pb, s.sbC, s.W + s.woff[k], s.bW[k], s.bW[k + 1]);
      __syncthreads();
      env_update_general<double, 0>(p, s, k, s.Cen, p.pb, s.sbC);
      if (tid == 0) {
        double *f = s.Fd;
        s.Fd = s.Fdn;
        s.Fdn = f;
      }
      __syncthreads();
    }
    if (tid == 0) {
      const double en = s.Fd[0];
      p.energy[w] = en / p.overlap[slot];
      p.ov_out[w] = p.overlap[slot];
      p.wt_out[w] = p.weight[slot];
    }
  }
}

#endif  // MQ_DEVICE_ONLY

}  // namespace mq
