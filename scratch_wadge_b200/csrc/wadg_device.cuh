// Device building blocks of the entropy-stable flux-differencing RHS:
// compile-time element sizes, FP64 reciprocal, log-mean, two-point EC flux,
// conservative <-> entropy variables.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace wadg {

// Element sizes of the reference's operator builder for cubature degree 2N
// (tri_cubature / tet_cubature tables of node_data.h as used by
// build_ref_ops_2D/3D, operators.cpp:104-341).
template <int DIM, int N> struct Sizes;
template <> struct Sizes<2, 1> { static constexpr int Np = 3,  Nq = 3,  Nfq = 2;  };
template <> struct Sizes<2, 2> { static constexpr int Np = 6,  Nq = 6,  Nfq = 3;  };
template <> struct Sizes<2, 3> { static constexpr int Np = 10, Nq = 12, Nfq = 4;  };
template <> struct Sizes<2, 4> { static constexpr int Np = 15, Nq = 16, Nfq = 5;  };
template <> struct Sizes<3, 1> { static constexpr int Np = 4,  Nq = 4,  Nfq = 3;  };
template <> struct Sizes<3, 2> { static constexpr int Np = 10, Nq = 11, Nfq = 6;  };
template <> struct Sizes<3, 3> { static constexpr int Np = 20, Nq = 23, Nfq = 12; };
template <> struct Sizes<3, 4> { static constexpr int Np = 35, Nq = 44, Nfq = 16; };

template <int DIM, int N> struct Elem {
  static constexpr int Nfaces = DIM + 1;
  static constexpr int Nq = Sizes<DIM, N>::Nq;
  static constexpr int Nfq = Sizes<DIM, N>::Nfq;
  static constexpr int NfqNf = Nfq * Nfaces;
  static constexpr int Nfields = DIM + 2;
  static constexpr int Nvgeo = DIM * DIM;
  static constexpr int Nfgeo = DIM + 1;
  static constexpr int NN = Nq + NfqNf;   // volume + face nodes
};

// an integer constant as a function argument
template <int V> struct IntTag {
  static constexpr int value = V;
};

// 8-byte asynchronous global -> shared copies (cp.async, sm_80 and later):
// the copies of a block are in flight together, occupying no registers, while
// the issuing threads go on computing; commit + wait completes them
__device__ __forceinline__ void cp_async8(double *dst_smem, const double *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// one 128-byte line on its way into L2
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}
// the lines of `bytes` bytes from p on, by threads t0, t0 + ts, ...
__device__ __forceinline__ void prefetch_lines(const void *p, int bytes, int t0, int ts) {
  for (int t = t0 * 128; t < bytes; t += ts * 128) prefetch_l2((const char *)p + t);
}

// Programmatic dependent launch: let the next kernel of the stream start its
// preamble, and wait for the previous one to finish (both do nothing in a
// kernel launched without the attribute).  What a predecessor writes may change
// while such a kernel already runs, so its pointers are neither const __restrict__
// nor read by __ldg: both promise data that is constant for the whole kernel,
// which lets a load take the non-coherent path or move above the wait
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

struct Phys {
  double gamma;
  double gm1;     // gamma - 1
  double cbeta;   // 1 / (2 (gamma - 1))
  double tau;     // LF penalty scale of the surface kernel
  double lgm1;    // log(gamma - 1)
  double igm1;    // 1 / (gamma - 1)
  double f1, f2;  // igm1 times the coefficients of polyF<0>
};

inline Phys make_phys(double gamma, double tau) {
  const double igm1 = 1.0 / (gamma - 1.0);
  return Phys{gamma, gamma - 1.0, 1.0 / (2.0 * (gamma - 1.0)), tau, log(gamma - 1.0), igm1,
              igm1 * 0.3333333333197528, igm1 * 0.20000278574597355};
}

// 1/x by one third-order step on the hardware estimate: with e = 1 - x y0,
// 1/x = y0 / (1 - e) = y0 (1 + e + e^2) + O(e^3).  The estimate
// rcp.approx.ftz.f64 is good to 1.0e-6 (measured over [1, 2), 7.6e8 points),
// so the remainder is below 1e-18: a rounding's worth of error in three FMAs,
// where two Newton-Raphson steps take four.  For the positive, normal-range
// arguments it is used on (sums of densities and inverse temperatures, log
// differences).
__device__ __forceinline__ double rcp_est(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rcp(double x) {
  const double y = rcp_est(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1/x with one Newton-Raphson step: relative error ~1e-12, for quantities
// that only feed a small series argument (the log-mean's u below 1.3e-5, where
// it moves the mean by less than 1e-17), never a result directly.  In the adjoint's
// pairs (pair_vjp) it also scales a derivative's smaller term, 2 G' f with f below
// 3.6e-3: 2.4e-15 of the derivative where the estimate is at its worst.  (The gradient's
// error against 64 bits is 1.1e-15 on the timed case; a third-order step there costs 0.9 %
// of the reverse sweep at 3D N=3, K=3072.)
__device__ __forceinline__ double rcp1(double x) {
  const double y = rcp_est(x);
  return fma(y, fma(-x, y, 1.0), y);
}

// Log-mean of a, b > 0: L(a, b) = (a - b) / (log a - log b).
//
// With s = a + b, f = (a - b) / s, u = f^2 and F(u) = atanh(f) / f =
// sum_k u^k / (2k+1): L = s / (2 F(u)) = s/2 G(u), 1/L = 2 F(u) / s.  The
// reference (Euler3Daffine.okl:43-71, Euler2D.okl:36-67) takes F's Taylor
// series below u = 1e-4 (3D) or 1e-3 (2D) and F = log(a/b) / (2f) above.  Here
// F and G = 1/F are polynomials in u over [0, logmean_u(T)], T = 0, 1, 2 by the
// range of u the caller has established: Chebyshev interpolants (the nearest
// singularity is u = 1, so a degree n falls as (4/b)^n on [0, b]), computed in
// 60 digits; relative error below 2e-17, 1.2e-17, 1.1e-17, less than a fifth of
// the sum's own rounding.  They reach the same accuracy as Taylor polynomials
// of degrees 2 (u < 4e-6), 4 (6e-4) and 12.  Beyond u = 6e-2 the difference of
// the per-node logarithms is at least 0.49; it carries the rounding of both (a
// unit in the last place each, 2.2e-16 |log|), so (a - b) / (log a - log b) is good to
// 4.5e-16 (|log a| + |log b|): 2e-15 for values within e^2 of 1, 1.3e-14 at 1e-6.
// Tests hold all of them to 1e-12 relative.
__host__ __device__ constexpr double logmean_u(int T) { return T == 0 ? 1.3e-5 : T == 1 ? 2e-3 : 6e-2; }
// the coefficients of F, highest degree first, all times c (c = 1 or a factor
// the caller wants in the product)
template <int T> __device__ __forceinline__ double polyF(double u) {
  if (T == 0) {
    return fma(fma(0.20000278574597355, u, 0.3333333333197528), u, 1.0);
  } else if (T == 1) {
    double p = 0.11156690948858601;
    p = fma(p, u, 0.14285634451046497);
    p = fma(p, u, 0.20000000057047174);
    p = fma(p, u, 0.3333333333331907);
    return fma(p, u, 1.0);
  } else {
    double p = 0.07530469258589562;
    p = fma(p, u, 0.06472373744008036);
    p = fma(p, u, 0.07704366316636192);
    p = fma(p, u, 0.0909047708631349);
    p = fma(p, u, 0.11111120157670987);
    p = fma(p, u, 0.1428571417961275);
    p = fma(p, u, 0.20000000000622098);
    p = fma(p, u, 0.3333333333333193);
    return fma(p, u, 1.0);
  }
}
template <int T> __device__ __forceinline__ double polyG(double u) {
  if (T == 0) {
    return fma(fma(-0.08888979683400786, u, -0.3333333333289071), u, 1.0);
  } else if (T == 1) {
    double p = -0.030303260937088336;
    p = fma(p, u, -0.046560655207755895);
    p = fma(p, u, -0.08888888902561856);
    p = fma(p, u, -0.3333333333332991);
    return fma(p, u, 1.0);
  } else {
    double p = -0.01416379152900634;
    p = fma(p, u, -0.01315451264187746);
    p = fma(p, u, -0.016809144823516215);
    p = fma(p, u, -0.021796030877831458);
    p = fma(p, u, -0.030194019711900843);
    p = fma(p, u, -0.04656084637107064);
    p = fma(p, u, -0.08888888889000143);
    p = fma(p, u, -0.3333333333333308);
    return fma(p, u, 1.0);
  }
}

// Per-node state of the two-point flux: everything of euler3d_flux /
// euler2d_flux (Euler3Daffine.okl:107-148, Euler2D.okl:139-161) that depends
// on one node only.
template <int DIM> struct NodeState {
  double rho, vel[DIM], beta;
};

// from conservative variables q; beta = rho / (2p)
// (Euler3Daffine.okl:22-26 pfun/beta, Euler2D.okl:19-21)
template <int DIM>
__device__ __forceinline__ NodeState<DIM> node_state(const double *q, const Phys &P) {
  NodeState<DIM> s;
  s.rho = q[0];
  const double ir = rcp(s.rho);
  double kin = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    s.vel[d] = q[1 + d] * ir;
    kin = fma(s.vel[d], s.vel[d], kin);
  }
  const double p = P.gm1 * (q[DIM + 1] - 0.5 * s.rho * kin);
  s.beta = 0.5 * s.rho * rcp(p);
  return s;
}

// sqrt(x) for x >= 1e-300, else 0 (the estimate takes a subnormal x for 0 and
// returns infinity; a speed below 1e-150 may count as none): one third-order step on the reciprocal
// square root estimate y0: with s0 = x y0 and e = 1 - s0 y0, sqrt(x) = s0 (1 -
// e)^(-1/2) = s0 (1 + e/2 + 3 e^2/8) + O(e^3), |e| < 1.9e-6 (measured
// over [1, 4)): at most 2.2e-16, in five operations.  For the surface kernels'
// wave speeds and U(V) at gamma = 1.4, where it enters every projected trace (the cases'
// errors against 64 bits are those of a correctly rounded square root)
__device__ __forceinline__ double fsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s = x * y;
  const double e = fma(-s, y, 1.0);
  return x >= 1e-300 ? fma(s * e, fma(e, 0.375, 0.5), s) : 0.0;
}

// conservative -> entropy variables (Euler3Daffine.okl:73-93 / Euler2D.okl:69-87)
template <int DIM>
__device__ __forceinline__ void VU(const double *U, double *V, const Phys &P) {
  const double rho = U[0], E = U[DIM + 1];
  double m2 = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) m2 = fma(U[1 + d], U[1 + d], m2);
  const double rhoe = E - 0.5 * m2 * rcp(rho);
  // s = log((gamma-1) rhoe / rho^gamma), written with two logarithms
  const double s = log(P.gm1 * rhoe) - P.gamma * log(rho);
  const double irhoe = rcp(rhoe);
  V[0] = (-E + rhoe * (P.gamma + 1.0 - s)) * irhoe;
#pragma unroll
  for (int d = 0; d < DIM; ++d) V[1 + d] = U[1 + d] * irhoe;
  V[DIM + 1] = -rho * irhoe;
}

// entropy -> conservative variables (Euler3Daffine.okl:95-105 / Euler2D.okl:89-98)
template <int DIM>
__device__ __forceinline__ void UV(const double *V, double *U, const Phys &P) {
  const double Vl = V[DIM + 1];
  double vv = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) vv = fma(V[1 + d], V[1 + d], vv);
  const double h = 0.5 * vv * rcp(Vl);  // vv / (2 V_l)
  const double sV = P.gamma - V[0] + h;
  // rhoe = ((gamma-1)/(-V_l)^gamma)^(1/(gamma-1)) exp(-sV/(gamma-1)), as one
  // exponential: exp((log(gamma-1) - gamma log(-V_l) - sV) / (gamma-1)).
  // For air (gamma = 1.4) the power is (-V_l)^(-7/2) = 1 / ((-V_l)^3
  // sqrt(-V_l)): a square root and a reciprocal in place of the logarithm
  // (within a few ulp of the general form)
  double rhoe;
  if (P.gamma == 1.4) {
    const double mv = -Vl;
    rhoe = exp((P.lgm1 - sV) * P.igm1) * rcp(mv * mv * mv * fsqrt(mv));
  } else {
    rhoe = exp((P.lgm1 - P.gamma * log(-Vl) - sV) * P.igm1);
  }
  U[0] = -rhoe * Vl;
#pragma unroll
  for (int d = 0; d < DIM; ++d) U[1 + d] = rhoe * V[1 + d];
  U[DIM + 1] = rhoe * (1.0 - h);
}

// Chandrashekar's entropy-conservative flux F_S(a, b), contracted with a
// direction n: the reference forms FxS, FyS, FzS and then FxS*nx + FyS*ny +
// FzS*nz (Euler3Daffine.okl:107-148, Euler2D.okl:139-161).  With rholog =
// L(rho), betalog = L(beta), ubar = (ua+ub)/2, pa = rhoavg / (2 betaavg), un = ubar.n:
//   F0 = rholog un, Fm = F0 ubar + pa n,
//   FE = (rholog (1/(2(gamma-1) betalog) + (ua.ub)/2) + pa) un,
// where ua.ub equals the reference's 2|ubar|^2 - avg(|u|^2).

// The largest u = ((a-b)/(a+b))^2, for the density and for beta, over every
// pair that a lane's element forms, volume-volume and volume-face: over the
// element's nodes it belongs to the extreme pair, ((max - min)/(max + min))^2.
// The extremes are taken of the high words (as integers: positive doubles sort
// as their bits do), with the low words that make u larger: high by up to 2e-6
// of max + min.  The L lanes of an element reduce by shuffles; node(n, rho,
// beta) gives the high words of node n's density and beta up to constant
// factors.  Infinite where a state is not positive or not finite.  Must be
// called by all 32 lanes of the warp.
template <int NN, int L, typename Node>
__device__ __forceinline__ double state_spread(int l, Node node) {
  int rmin, rmax, bmin, bmax;
  node(l < NN ? l : 0, rmin, bmin);
  rmax = rmin;
  bmax = bmin;
#pragma unroll 4
  for (int n = l + L; n < NN; n += L) {
    int r, b;
    node(n, r, b);
    rmin = min(rmin, r);
    rmax = max(rmax, r);
    bmin = min(bmin, b);
    bmax = max(bmax, b);
  }
#pragma unroll
  for (int o = L / 2; o >= 1; o >>= 1) {
    rmin = min(rmin, __shfl_xor_sync(0xffffffffu, rmin, o));
    rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    bmin = min(bmin, __shfl_xor_sync(0xffffffffu, bmin, o));
    bmax = max(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
  }
  // sign bit: not positive (as an integer, below every positive high word);
  // exponent all ones: infinite or NaN
  if (rmin <= 0 || bmin <= 0 || rmax >= 0x7ff00000 || bmax >= 0x7ff00000) return INFINITY;
  const double r0 = __hiloint2double(rmin, 0), r1 = __hiloint2double(rmax, -1);
  const double b0 = __hiloint2double(bmin, 0), b1 = __hiloint2double(bmax, -1);
  const double fr = (r1 - r0) * rcp(r1 + r0), fb = (b1 - b0) * rcp(b1 + b0);
  return fmax(fr * fr, fb * fb);
}

// The T of the log-mean's polynomials that holds for every pair of the warp's
// elements (u < logmean_u(T)), or 3 when none does.  The pair loops then carry
// no per-pair vote or branch.  Share of the warps with T = 0 / 1 / 2 / 3:
// Taylor-Green at Mach 0.1 on 24576 tets all 0; at Mach 0.3, N=4, K=4374 0 / 1
// / 0 / 0; 2D vortex K=2048 .93 / .04 / .03 / 0; density wave on 10368 warped
// tets 0 / .06 / .94 / 0.
template <int NN, int L, typename Node>
__device__ __forceinline__ int state_range(int l, Node node) {
  const double u = state_spread<NN, L>(l, node);
  int t = 3;
#pragma unroll
  for (int T = 2; T >= 0; --T)
    if (__all_sync(0xffffffffu, u < logmean_u(T))) t = T;
  return t;
}

// The means of R row states (density halved, beta and, for T = 3, their
// logarithms) against one column state: rl = L(rho), pa = rhoavg / (2 betaavg)
// and 1/(2(gamma-1) L(beta)) as the product ib pf.  T: the range of u
// (state_range).  T = 3 takes the polynomials of T = 2 where every lane's pairs
// allow it (a warp vote per column), else per pair the polynomial or the
// log-difference.  R independent chains in one basic block, which the scheduler
// interleaves.  Must be called by all 32 lanes of the warp.
template <int R, int T>
__device__ __forceinline__ void pair_means(const double (&ahr)[R], const double (&ab)[R],
                                           const double (&alr)[R], const double (&alb)[R],
                                           double bhr, double bb, double blr, double blb,
                                           const Phys &P, double (&rl)[R], double (&pa)[R],
                                           double (&ib)[R], double (&pf)[R]) {
  constexpr int TP = T < 2 ? T : 2;
  double ur[R], ub[R], sr[R], dr[R], db[R], isb[R];
  bool near = true;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    sr[r] = ahr[r] + bhr;  // the average density
    dr[r] = ahr[r] - bhr;
    db[r] = ab[r] - bb;
    // 1/(a+b) of the densities only forms u: one Newton step where u is small
    const double isr = T == 0 ? rcp1(sr[r]) : rcp(sr[r]);
    isb[r] = rcp(ab[r] + bb);
    const double fr = dr[r] * isr, fb = db[r] * isb[r];
    ur[r] = fr * fr;
    ub[r] = fb * fb;
    pa[r] = sr[r] * isb[r];
    if (T == 3) near = near && fmax(ur[r], ub[r]) < logmean_u(2);
  }
  if (T < 3 || __all_sync(0xffffffffu, near)) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rl[r] = sr[r] * polyG<TP>(ur[r]);
      if (T == 0) {  // the factor 1/(gamma-1) in the coefficients
        ib[r] = isb[r];
        pf[r] = fma(fma(P.f2, ub[r], P.f1), ub[r], P.igm1);
      } else {
        ib[r] = isb[r] * P.igm1;
        pf[r] = polyF<TP>(ub[r]);
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      rl[r] = ur[r] < logmean_u(2) ? sr[r] * polyG<2>(ur[r]) : 2.0 * dr[r] * rcp(alr[r] - blr);
      ib[r] = ub[r] < logmean_u(2) ? isb[r] * P.igm1 : (alb[r] - blb) * P.cbeta;
      pf[r] = ub[r] < logmean_u(2) ? polyF<2>(ub[r]) : rcp(db[r]);
    }
  }
}

// Two-point flux F_S(a, b).n for states without precomputed logarithms (surface
// traces): beyond the series range the log-mean evaluates log(a/b) itself, as
// the reference does.  WARP: called by all 32 lanes, which take the short
// polynomials where all their pairs allow it (traces of a smooth flow differ
// little across a face)
template <int DIM, bool WARP = false>
__device__ __forceinline__ void ecflux_n_nolog(const NodeState<DIM> &a, const NodeState<DIM> &b,
                                               const double *n, const Phys &P, double *F) {
  const double hs = 0.5 * (a.rho + b.rho), dr = a.rho - b.rho;
  const double sb = a.beta + b.beta, db = a.beta - b.beta;
  const double isr = rcp(hs), isb = rcp(sb);
  const double fr = 0.5 * dr * isr, fb = db * isb;
  const double ur = fr * fr, ub = fb * fb;
  double rl, ib;  // L(rho), 1/(2(gamma-1) L(beta))
  if (WARP && __all_sync(0xffffffffu, fmax(ur, ub) < logmean_u(0))) {
    rl = hs * polyG<0>(ur);
    ib = isb * fma(fma(P.f2, ub, P.f1), ub, P.igm1);
  } else {
    rl = ur < logmean_u(2) ? hs * polyG<2>(ur) : dr / log(a.rho / b.rho);
    ib = ub < logmean_u(2) ? isb * P.igm1 * polyF<2>(ub) : P.cbeta * (log(a.beta / b.beta) / db);
  }
  const double pa = hs * isb;
  double ub2[DIM], un = 0.0, vv = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    ub2[d] = 0.5 * (a.vel[d] + b.vel[d]);
    un = fma(ub2[d], n[d], un);
    vv = fma(a.vel[d], b.vel[d], vv);
  }
  const double f4 = fma(rl, fma(0.5, vv, ib), pa);
  const double F0 = rl * un;
  F[0] = F0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) F[1 + d] = fma(F0, ub2[d], pa * n[d]);
  F[DIM + 1] = f4 * un;
}

// node state of a conservative trace without the logarithms (for
// ecflux_n_nolog), with |u|^2 and the squared sound speed gamma p / rho of the
// surface penalty; reciprocals (rcp) in place of divisions
template <int DIM>
__device__ __forceinline__ NodeState<DIM> node_state_surf(const double *q, int stride, const Phys &P,
                                                          double &kin, double &c2) {
  NodeState<DIM> s;
  s.rho = q[0];
  const double ir = rcp(s.rho);
  kin = 0.0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    s.vel[d] = q[(1 + d) * stride] * ir;
    kin = fma(s.vel[d], s.vel[d], kin);
  }
  const double p = P.gm1 * (q[(DIM + 1) * stride] - 0.5 * s.rho * kin);
  s.beta = 0.5 * s.rho * rcp(p);
  c2 = P.gamma * p * ir;
  return s;
}

}  // namespace wadg
