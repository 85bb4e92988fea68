// Pair-scheduled volume kernel (the default volume kernel) and the fused
// stage kernel built on it.
//
// The reference's volume kernels (one thread per row, Euler3Daffine.okl:152-417),
// organised so that every volume-face pair (i, f) is evaluated once: F_S(u_i, uf_f).nJ_f feeds both
// the volume row i (weight 1/2 VqLq_if) and the face row f (weight
// -1/2 VfPq_fi).  The reference evaluates it twice, once per row
// (Euler3Daffine.okl:327-362 and :387-406); the flux is symmetric in its two
// states, so the sums are the same.
//
// The FP64 pipe bounds these kernels (two cycles per warp instruction and SM
// quarter; DMMA shares it: 34.5 TFLOP/s of FMAs alone, 36.7 of DMMAs alone, 32
// to 35 of both together), so the pair loops do only what depends on both
// nodes.  With h = u/2 per node:
//   * un = (h_i + h_j).n.  Affine elements: volume pairs take n = G^T D_ij, so
//     un = sum_a D^a_ij (U^a_i + U^a_j) from the nodes' contravariant velocities
//     U = G h; volume-face pairs of one face share n, so un = h_i.n + h_f.n,
//     the first once per row and face, the second once per face node.
//   * sums over j instead of terms (affine): sum_j F0 (h_i + h_j) = h_i sum_j F0 + sum_j F0 h_j;
//     sum_j pa n = G^T sum_j pa D_ij, or n sum_f pa over one face; the kinetic
//     part of the energy flux, F0 (u_i.u_j)/2, sums to 2 h_i.(sum_j F0 h_j).
//     The same sums serve the face rows, with i and f exchanged.
//   * curved elements: a face node keeps n_f = sum_a nr_a G^a_f, a row
//     n_i = sum_a nr_a G^a_i per face, and a pair's direction is their sum.
// FP64 instructions per volume / volume-face pair (3D, nearly equal states):
// affine 56 / 54 -> 36 / 40.  Measured (the terms pair by pair before): volume +
// surface 0.250 -> 0.219 ms (Taylor-Green, N=3, K=24576), 0.073 -> 0.063 ms (2D
// vortex, N=3, K=32768); volume 0.548 -> 0.330 ms (curved N=4, K=10368, where the
// wider log-mean polynomials replace the logarithms too).
//
// Layout.  A group of L lanes owns one element; lane l owns the R volume rows
// i = l + L*r (register accumulators; the padding row, if any, computes on a
// clamped index and is never stored).  Two warps share each group of G = 32/L
// elements (one where a half of the face nodes would be fewer than L): each
// walks its own volume columns and its own face nodes.  The face nodes come in
// blocks: the warp's faces one after another where a face has at least L nodes
// or the warps take one face each (FACES), else all of the warp's face nodes as one block.  At step s of a block
// of n nodes lane l takes node (l + s) mod n, so the L lanes of a group always
// touch L distinct face rows, and the two warps never the same one: both add
// their R contributions to one copy of the face-row accumulators in shared
// memory, a __syncwarp between steps ordering the read-modify-writes.  The
// schedule is fixed, so results are deterministic (no atomics).  Warps stay
// converged throughout so that pair_means can vote on the log-mean branch.
//
// Persistent CTAs: operator tables are staged in shared memory once per CTA;
// the face weights in a rotated layout [node][r][l] so that the lanes of a step
// read consecutive words.  In the volume kernel's batch loop the warps of an
// element group synchronise only among themselves (named barriers): a
// group's shared memory is its own, so no group waits for another.
#pragma once

#include "wadg_device.cuh"

namespace wadg {

// Node-to-thread map: L lanes per element, R rows per lane.  RR = 0: about
// three rows per lane (L = the power of two >= Nq/3); RR > 0: about RR rows
// (an autotuner candidate where it pads less, e.g. 2D N=4: Nq = 16 fills
// L = 4 x 4 or 8 x 2 exactly, against 8 x 3 = 24 slots by default)
// HH = 0: two warps per element group, or one; HH = Nfaces: a warp per face.
template <int DIM, int N, int RR = 0, int HH = 0> struct VolTile {
  using El = Elem<DIM, N>;
  static constexpr int Lraw = RR > 0 ? (El::Nq + RR - 1) / RR : (El::Nq + 2) / 3;
  static constexpr int L = Lraw <= 1 ? 1 : Lraw <= 2 ? 2 : Lraw <= 4 ? 4 : Lraw <= 8 ? 8 : Lraw <= 16 ? 16 : 32;
  static constexpr int R = (El::Nq + L - 1) / L;
  static constexpr int G = 32 / L;  // elements per warp group
  static_assert(El::NfqNf >= L, "face schedule needs NfqNf >= L");
  static constexpr bool FACES = El::Nfq >= L || HH;  // blocks of one face
  // steps of a block: a face of fewer nodes than lanes (2D N=4 with a warp per
  // face) leaves the lanes past its end idle
  static constexpr int NR = El::Nfq > L ? El::Nfq : L;
  static constexpr int NP = FACES ? El::Nfaces * NR : El::NfqNf;  // (step, lane) pairs / L of all blocks
  static constexpr int H = HH ? HH : El::NfqNf / 2 >= L ? 2 : 1;  // warps per element group
  static_assert(HH == 0 || HH == El::Nfaces, "a warp per face, or the default");
  // the face nodes [f0(h), f0(h + 1)) of warp h: whole faces where a block is one
  __host__ __device__ static constexpr int f0(int h) {
    return FACES ? (h * El::Nfaces + H - 1) / H * El::Nfq : (h * El::NfqNf + H - 1) / H;
  }
  __host__ __device__ static constexpr int nf(int h) { return f0(h + 1) - f0(h); }
  // the volume columns [c0(h), c0(h + 1)): so that the warps take about as many steps each
  __host__ __device__ static constexpr int c0(int h) {
    const int c = h * (El::Nq + NP) / H - (FACES ? f0(h) / El::Nfq * NR : f0(h));
    return c < 0 ? 0 : c > El::Nq ? El::Nq : c;
  }
};

template <int DIM, int N, bool CURVED, int W, int RR = 0, int HH = 0>
struct VolPairsCfg {
  using El = Elem<DIM, N>;
  using T = VolTile<DIM, N, RR, HH>;
  static constexpr int H = T::H;                      // warps per element group
  static constexpr int threads = 32 * W;
  static constexpr int E = (W / H) * T::G;            // elements of a CTA's groups
  // elements per batch of a work list (with a warp per face the CTA's warps follow the
  // mesh's size, the batch does not)
  static constexpr int EB = HH ? 12 / HH * T::G : E;
  // one direction per block and the sums of the header comment
  static constexpr bool SPLIT = !CURVED && T::FACES;
  // an element's state block (doubles; [2]: double2): logarithms [2][NN] |
  // rho/2, beta [2][NN] | h0, h1 [2][NN] | 3D: h2 (SPLIT: and h.n of a face node, U^0 of a
  // volume node) | SPLIT: the rest of U [2][Nq], 2D: h.n of the face nodes [NF] |
  // curved: G/2 of the volume nodes [Nvgeo][Nq], n_f of the face nodes [DIM][NF]
  static constexpr int oA = 2 * El::NN, oB = 4 * El::NN, oC = 6 * El::NN;
  static constexpr int oD = oC + (DIM == 3 ? (SPLIT ? 2 : 1) * El::NN : 0);
  static constexpr int oX = oD + (SPLIT ? 2 * El::Nq : 0);
  static constexpr int oG = oX + (SPLIT && DIM == 2 ? El::NfqNf : 0);
  static constexpr int oN = oG + (CURVED ? El::Nvgeo * El::Nq : 0);
  static constexpr int nS = oN + (CURVED ? DIM * El::NfqNf : 0);
  // the element strides are 2L mod 16 (the state block, read as double2 by a
  // quarter warp at a time) or L mod 16 (single words, by a half warp), so that
  // neighbouring elements' lanes fall into different banks
  static constexpr int up(int x, int m) { return x % 16 == m % 16 ? x : up(x + 1, m); }
  static constexpr int mL = T::L < 8 ? T::L : 8;
  static constexpr int mx(int a, int b) { return a > b ? a : b; }
  // the state block of an element is reused after the pair phase for the
  // update's staging arrays (3 x Nfields x Nq)
  static constexpr int SE = up(mx(nS, 3 * El::Nfields * El::Nq), mL < 8 ? 2 * mL : 8);
  // face-row accumulators: SPLIT [2][NF] (sum F0, sum pa), (m0, m1), 3D (m2, E), 2D E [NF];
  // else the Nfields rows [NF]
  static constexpr int nA = (DIM == 3 ? 6 : 5) * El::NfqNf;
  // (-2 mod 16 serves L = 1 as well as 2, and 16 warps of 2D N=1 fit with it)
  static constexpr int SA = !SPLIT ? up(El::Nfields * El::NfqNf, mL)
                            : T::L == 1 && nA % 16 == 14 ? nA : up(nA, mL < 8 ? 2 * mL : 8);
  // per-face nJ and G (affine), and the next slice's G
  static constexpr int SN = CURVED ? 0 : El::Nfaces * DIM + 2 * El::Nvgeo;
  static constexpr int nD = DIM * El::Nq * El::Nq;
  static constexpr int nW = T::R * T::NP * T::L;
  static constexpr size_t fixed = sizeof(double) * (size_t)(nD + 2 * nW + El::Nfaces * DIM);
  static constexpr size_t per_elem = sizeof(double) * (size_t)(SE + SA + SN);
  static constexpr size_t smem = fixed + E * per_elem;
  // the volume kernel stages the next batch's face traces (cp.async) while it
  // computes the current one, where shared memory has room for them
  static constexpr size_t pre = sizeof(double) * (size_t)E * El::Nfields * El::NfqNf;
  static constexpr bool PREFETCH = smem + pre <= 227 * 1024;
  static constexpr size_t smem_vol = smem + (PREFETCH ? pre : 0);
};

// Shared-memory carve-up and the phases common to the kernels.
template <int DIM, int N, bool CURVED, int W, int RR = 0, int HH = 0>
struct VolPairs {
  using El = Elem<DIM, N>;
  using T = VolTile<DIM, N, RR, HH>;
  using C = VolPairsCfg<DIM, N, CURVED, W, RR, HH>;
  static constexpr int Nq = El::Nq, NF = El::NfqNf, Nfq = El::Nfq, NN = El::NN;
  static constexpr int Nf = El::Nfields, NG = El::Nvgeo, L = T::L, R = T::R, G = T::G, E = C::E;
  static constexpr int SE = C::SE, SA = C::SA, SN = C::SN, H = C::H;
  static constexpr bool SPLIT = C::SPLIT, FACES = T::FACES;
  static_assert(SE % 2 == 0 && (!SPLIT || SA % 2 == 0), "double2 blocks");

  double *sD, *sW, *sD2, *sNr, *sSt, *sAcc, *sNrm, *sPre;
  int tid, h, g, l, e;

  __device__ __forceinline__ VolPairs(double *smem) {
    sD = smem;                          // (Drq, Dsq) [2][j][i]
    sW = sD + 2 * Nq * Nq;              // [2][block][step][R][L] 1/2 VqLq(i, f), -1/2 VfPq(f, i); 0 on padding rows
    sSt = sW + 2 * C::nW;               // [E][SE]     node states
    sAcc = sSt + E * SE;                // [E][SA]     face-row accumulators
    sD2 = sAcc + E * SA;                // Dtq [j][i]  (3D)
    sNr = sD2 + (DIM - 2) * Nq * Nq;    // reference normals [Nfaces][DIM]
    sNrm = sNr + El::Nfaces * DIM;      // [E][SN]     per-face nJ, G, the next slice's G (affine)
    sPre = sNrm + E * SN;               // [E][Nf][NF] staged face traces (volume kernel, PREFETCH)
    tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    h = warp % H;
    g = lane / L;
    l = lane % L;
    e = (warp / H) * G + g;
  }

  // steps of the block at face node fb, and the node that lane l takes at step s
  // (past a face's end: its last node, with weights 0 and no addition)
  static constexpr bool IDLE = FACES && Nfq < L;
  __device__ static __forceinline__ int steps(int h) { return FACES ? T::NR : T::nf(h); }
  __device__ static __forceinline__ int node(int l, int s, int n) {
    const int ff = l + s;
    return ff >= n ? ff - n : ff;
  }
  __device__ static __forceinline__ int weights(int fb) {
    return (FACES ? fb / Nfq * T::NR : fb) * R * L;
  }

  __device__ __forceinline__ void load_tables(const double *nrJ, const double *nsJ,
                                              const double *ntJ, const double *Drq,
                                              const double *Dsq, const double *Dtq,
                                              const double *VqLq, const double *VfPq) {
#pragma unroll 4
    for (int t = tid; t < Nq * Nq; t += C::threads) {
      sD[2 * t] = Drq[t];
      sD[2 * t + 1] = Dsq[t];
      if (DIM == 3) sD2[t] = Dtq[t];
    }
#pragma unroll 4
    for (int t = tid; t < C::nW; t += C::threads) {
      const int ll = t % L, r = (t / L) % R, p = t / (L * R);
      const int hh = !FACES && H == 2 && p >= T::f0(1);
      const int fb = FACES ? p / T::NR * Nfq : T::f0(hh);
      const int i = ll + L * r, ff = node(ll, FACES ? p % T::NR : p - fb, steps(hh)), f = fb + ff;
      const bool on = i < Nq && (!IDLE || ff < Nfq);
      sW[2 * t] = on ? 0.5 * VqLq[i + f * Nq] : 0.0;
      sW[2 * t + 1] = on ? -0.5 * VfPq[f + i * NF] : 0.0;
    }
    for (int t = tid; t < El::Nfaces; t += C::threads) {
      sNr[t * DIM + 0] = nrJ[t * Nfq];
      sNr[t * DIM + 1] = nsJ[t * Nfq];
      if (DIM == 3) sNr[t * DIM + 2] = ntJ[t * Nfq];
    }
  }

  // affine: the geometric factors (constant per element, read at node 0 as
  // Euler3Daffine.okl:205) of the slice whose first element is k0 + e0, into the next
  // slice's slots (asynchronous copies; the prologue reads them)
  __device__ __forceinline__ void fetch_geo(int K, int k0, int e0, int t0, int ts,
                                            const double *vgeo) const {
    if (CURVED) return;
    for (int t = t0; t < G * NG; t += ts) {
      const int ee = e0 + t / NG, c = t % NG;
      const int k = min(k0 + ee, K - 1);
      cp_async8(sNrm + ee * SN + El::Nfaces * DIM + NG + c, vgeo + (size_t)k * Nq * NG + c * Nq);
    }
  }

  // Node states of one element group's batch elements [e0, e0 + G), by TS
  // threads t0, t0 + TS, ...; elements past the end replicate the last
  // element so that every lane computes on valid data.  ufs: the group's
  // face traces already staged in shared memory, or null.  The states carry
  // no logarithms (fill_logs adds them where a group needs
  // them).  The loads of a thread's nodes (global for the volume nodes) are
  // issued before their node states are computed
  template <int TS>
  __device__ __forceinline__ void prologue_group(int K, int k0, int e0, int t0, const double *vgeo,
                                                 const double *vfgeo, const double *uq,
                                                 const double *uf, const Phys &P,
                                                 const double *ufs) {
    constexpr int NT = (G * NN + TS - 1) / TS;
    // the thread's nodes in chunks of CH, a chunk's loads all in flight: up to
    // five nodes at once, more four at a time
    constexpr int CH = NT <= 5 ? NT : 4;
#pragma unroll 1
    for (int c0 = 0; c0 < NT; c0 += CH) {
      double u[CH][Nf];
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int t = t0 + (c0 + j) * TS;
        if (c0 + j < NT && t < G * NN) {
          const int ee = e0 + t / NN, n = t % NN;
          const int k = min(k0 + ee, K - 1);
          // staged traces only for the group's own elements (a clamped
          // element's copy may sit in another group's range)
          const int kk = k - k0;
          const double *fsrc = (ufs && kk >= e0 && kk < e0 + G) ? ufs + (size_t)kk * NF * Nf
                                                               : uf + (size_t)k * NF * Nf;
          const double *src = (n < Nq) ? uq + (size_t)k * Nq * Nf + n : fsrc + (n - Nq);
          const int stride = (n < Nq) ? Nq : NF;
#pragma unroll
          for (int f = 0; f < Nf; ++f) u[j][f] = src[f * stride];
        } else {
#pragma unroll
          for (int f = 0; f < Nf; ++f) u[j][f] = 1.0;
        }
      }
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int t = t0 + (c0 + j) * TS;
        if (c0 + j < NT && t < G * NN) {
          const int ee = e0 + t / NN, n = t % NN;
          const int k = min(k0 + ee, K - 1);
          const NodeState<DIM> s = node_state<DIM>(u[j], P);
          double *st = sSt + ee * SE;
          double hv[DIM];
#pragma unroll
          for (int d = 0; d < DIM; ++d) hv[d] = 0.5 * s.vel[d];
          ((double2 *)(st + C::oA))[n] = make_double2(0.5 * s.rho, s.beta);
          ((double2 *)(st + C::oB))[n] = make_double2(hv[0], hv[1]);
          if (SPLIT) {
            // contravariant velocity (volume node) or h.n (face node; n = G^T nr of its face)
            const double *Gk = sNrm + ee * SN + El::Nfaces * DIM + NG;
            double U[DIM];
#pragma unroll
            for (int a = 0; a < DIM; ++a) {
              U[a] = 0.0;
#pragma unroll
              for (int d = 0; d < DIM; ++d) U[a] = fma(Gk[a * DIM + d], hv[d], U[a]);
            }
            double x = U[0];
            if (n >= Nq) {
              const double *nr = sNr + (n - Nq) / Nfq * DIM;
              x = 0.0;
#pragma unroll
              for (int a = 0; a < DIM; ++a) x = fma(nr[a], U[a], x);
            }
            if (DIM == 3) {
              ((double2 *)(st + C::oC))[n] = make_double2(hv[DIM - 1], x);
              if (n < Nq) ((double2 *)(st + C::oD))[n] = make_double2(U[1], U[DIM - 1]);
            } else if (n < Nq) {
              ((double2 *)(st + C::oD))[n] = make_double2(U[0], U[1]);
            } else {
              st[C::oX + n - Nq] = x;
            }
          } else if (DIM == 3) {
            st[C::oC + n] = hv[DIM - 1];
          }
          if (CURVED) {  // geometric factors stored halved: a pair's average
                         // (G_i + G_j)/2 is then one addition, with the same bits
            if (n < Nq) {
#pragma unroll
              for (int c = 0; c < NG; ++c)
                st[C::oG + c * Nq + n] = 0.5 * vgeo[(size_t)k * Nq * NG + c * Nq + n];
            } else {
              const double *gf = vfgeo + (size_t)k * NF * NG + (n - Nq);
              const double *nr = sNr + (n - Nq) / Nfq * DIM;
#pragma unroll
              for (int d = 0; d < DIM; ++d) {
                double v = 0.0;
#pragma unroll
                for (int a = 0; a < DIM; ++a) v = fma(gf[(a * DIM + d) * NF], nr[a], v);
                st[C::oN + d * NF + n - Nq] = 0.5 * v;
              }
            }
          }
        }
      }
    }
    for (int t = t0; t < G * SA; t += TS) sAcc[e0 * SA + t] = 0.0;
    if (!CURVED) {
      for (int t = t0; t < G * (El::Nfaces + 1); t += TS) {
        double *nm = sNrm + (e0 + t / (El::Nfaces + 1)) * SN;
        const int fc = t % (El::Nfaces + 1);
        const double *Gk = nm + El::Nfaces * DIM + NG;
        if (fc == El::Nfaces) {
#pragma unroll
          for (int c = 0; c < NG; ++c) nm[El::Nfaces * DIM + c] = Gk[c];
        } else {
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            double v = 0.0;
#pragma unroll
            for (int a = 0; a < DIM; ++a) v = fma(Gk[a * DIM + d], sNr[fc * DIM + a], v);
            nm[fc * DIM + d] = v;
          }
        }
      }
    }
  }

  // a node's state as the pair phase keeps it: density and velocity halved
  struct Node {
    double hr, b, h[DIM], x, lr, lb;
  };
  template <int TT>
  __device__ __forceinline__ Node load(const double *st, int n) const {
    Node s;
    const double2 a = ((const double2 *)(st + C::oA))[n], b = ((const double2 *)(st + C::oB))[n];
    s.hr = a.x;
    s.b = a.y;
    s.h[0] = b.x;
    s.h[1] = b.y;
    s.x = 0.0;
    if (DIM == 3) {
      if (SPLIT) {
        const double2 c = ((const double2 *)(st + C::oC))[n];
        s.h[DIM - 1] = c.x;
        s.x = c.y;
      } else {
        s.h[DIM - 1] = st[C::oC + n];
      }
    }
    s.lr = s.lb = 0.0;
    if (TT == 3) {
      const double2 c = ((const double2 *)st)[n];
      s.lr = c.x;
      s.lb = c.y;
    }
    return s;
  }

  // all flux pairs of element e: this warp's volume columns and face nodes;
  // the rows into F (registers), the face rows into the element's face
  // accumulators (SPLIT: the sums that face_row combines).  TT: the range of
  // the states (state_range).
  template <int TT>
  __device__ __forceinline__ void pairs(double (&F)[R][Nf], const Phys &P) const {
    const double *st = sSt + e * SE;
    double *acc_f = sAcc + e * SA;
    double ahr[R], ab[R], alr[R], alb[R], ah[R][DIM];
    double a0[R], am[R][DIM], ap[R][DIM], aE[R];  // sums of F0, F0 h_j (else Fm), pa n, FE
    int ir[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      ir[r] = min(l + L * r, Nq - 1);  // padding row computes on a clamped index
      const Node s = load<TT>(st, ir[r]);
      ahr[r] = s.hr;
      ab[r] = s.b;
      alr[r] = s.lr;
      alb[r] = s.lb;
      a0[r] = aE[r] = 0.0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        ah[r][d] = s.h[d];
        am[r][d] = ap[r][d] = 0.0;
      }
    }
    double rl[R], pa[R], ib[R], pf[R];

    // volume-volume pairs
    {
      double U[R][DIM], Ge[NG];
      if (SPLIT) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double2 u = ((const double2 *)(st + C::oD))[ir[r]];
          if (DIM == 3) U[r][0] = st[C::oC + 2 * ir[r] + 1];
          U[r][DIM - 2] = u.x;
          U[r][DIM - 1] = u.y;
        }
      } else if (!CURVED) {
#pragma unroll
        for (int c = 0; c < NG; ++c) Ge[c] = sNrm[e * SN + El::Nfaces * DIM + c];
      }
      for (int j = T::c0(h); j < T::c0(h + 1); ++j) {
        const Node B = load<TT>(st, j);
        double UB[DIM];
        if (SPLIT) {
          const double2 u = ((const double2 *)(st + C::oD))[j];
          if (DIM == 3) UB[0] = B.x;
          UB[DIM - 2] = u.x;
          UB[DIM - 1] = u.y;
        }
        pair_means<R, TT>(ahr, ab, alr, alb, B.hr, B.b, B.lr, B.lb, P, rl, pa, ib, pf);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          double D[DIM];
          const double2 d2 = ((const double2 *)sD)[ir[r] + j * Nq];
          D[0] = d2.x;
          D[1] = d2.y;
          if (DIM == 3) D[DIM - 1] = sD2[ir[r] + j * Nq];
          if (SPLIT) {
            double un = 0.0;
#pragma unroll
            for (int a = 0; a < DIM; ++a) un = a ? fma(D[a], U[r][a] + UB[a], un) : D[a] * (U[r][a] + UB[a]);
            const double F0 = rl[r] * un;
            a0[r] += F0;
            aE[r] = fma(fma(rl[r], ib[r] * pf[r], pa[r]), un, aE[r]);
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              am[r][d] = fma(F0, B.h[d], am[r][d]);
              ap[r][d] = fma(pa[r], D[d], ap[r][d]);  // contravariant
            }
          } else {
            double nv[DIM], ub[DIM], un = 0.0, hv = 0.0;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              nv[d] = 0.0;
#pragma unroll
              for (int a = 0; a < DIM; ++a) {
                const double gad = CURVED ? st[C::oG + (a * DIM + d) * Nq + ir[r]] +
                                                st[C::oG + (a * DIM + d) * Nq + j]
                                          : Ge[a * DIM + d];
                nv[d] = a ? fma(gad, D[a], nv[d]) : gad * D[a];
              }
              ub[d] = ah[r][d] + B.h[d];
              un = d ? fma(ub[d], nv[d], un) : ub[d] * nv[d];
              hv = d ? fma(2.0 * ah[r][d], B.h[d], hv) : 2.0 * ah[r][d] * B.h[d];
            }
            const double F0 = rl[r] * un;
            a0[r] += F0;
            aE[r] = fma(fma(rl[r], fma(ib[r], pf[r], hv), pa[r]), un, aE[r]);
#pragma unroll
            for (int d = 0; d < DIM; ++d) am[r][d] = fma(F0, ub[d], fma(pa[r], nv[d], am[r][d]));
          }
        }
      }
      if (SPLIT) {  // sum pa n = G^T (contravariant sum)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          double v[DIM];
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            v[d] = 0.0;
#pragma unroll
            for (int a = 0; a < DIM; ++a)
              v[d] = fma(sNrm[e * SN + El::Nfaces * DIM + a * DIM + d], ap[r][a], v[d]);
          }
#pragma unroll
          for (int d = 0; d < DIM; ++d) ap[r][d] = v[d];
        }
      }
    }

    // volume-face pairs, each evaluated once: warp h takes its face nodes
#pragma unroll 1
    for (int fb = T::f0(h); fb < T::f0(h) + T::nf(h); fb += FACES ? Nfq : NF) {
      const int n = steps(h);
      // per block (one face): the direction, or the row's part of it
      double nb[DIM], xi[R], nr[R][DIM], pb[R];
      if (SPLIT) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) nb[d] = sNrm[e * SN + fb / Nfq * DIM + d];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          pb[r] = xi[r] = 0.0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) xi[r] = d ? fma(ah[r][d], nb[d], xi[r]) : ah[r][d] * nb[d];
        }
      } else if (CURVED && FACES) {
        row_normals(st, ir, fb / Nfq, nr);
      }
      const double2 *wb = (const double2 *)sW + weights(fb) + l;
#pragma unroll 1
      for (int s = 0; s < n; ++s) {
        const int ff = node(l, s, n), f = fb + (IDLE ? min(ff, Nfq - 1) : ff);
        const bool on = !IDLE || ff < Nfq;
        const Node B = load<TT>(st, Nq + f);
        pair_means<R, TT>(ahr, ab, alr, alb, B.hr, B.b, B.lr, B.lb, P, rl, pa, ib, pf);
        if (SPLIT) {
          const double x = DIM == 3 ? B.x : st[C::oX + f];
          double g0, gp, gE, gm[DIM];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double2 w = wb[(s * R + r) * L];
            const double un = xi[r] + x, F0 = rl[r] * un;
            const double f4u = fma(rl[r], ib[r] * pf[r], pa[r]) * un;
            const double g1 = w.x * F0, g2 = w.y * F0;
            a0[r] += g1;
            pb[r] = fma(w.x, pa[r], pb[r]);
            aE[r] = fma(w.x, f4u, aE[r]);
            g0 = r ? g0 + g2 : g2;
            gp = r ? fma(w.y, pa[r], gp) : w.y * pa[r];
            gE = r ? fma(w.y, f4u, gE) : w.y * f4u;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              am[r][d] = fma(g1, B.h[d], am[r][d]);
              gm[d] = r ? fma(g2, ah[r][d], gm[d]) : g2 * ah[r][d];
            }
          }
          if (on) {
            double2 *q = (double2 *)acc_f + f;
            const double2 q0 = q[0], q1 = q[NF];
            if (DIM == 3) {
              const double2 q2 = q[2 * NF];
              q[2 * NF] = make_double2(q2.x + gm[DIM - 1], q2.y + gE);
            } else {
              acc_f[4 * NF + f] += gE;
            }
            q[0] = make_double2(q0.x + g0, q0.y + gp);
            q[NF] = make_double2(q1.x + gm[0], q1.y + gm[1]);
          }
        } else {
          double af[Nf], nfv[DIM];
          if (!FACES && CURVED) row_normals(st, ir, f / Nfq, nr);
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            nfv[d] = CURVED ? st[C::oN + d * NF + f] : sNrm[e * SN + f / Nfq * DIM + d];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const double2 w = wb[(s * R + r) * L];
            double nv[DIM], ub[DIM], un = 0.0, hv = 0.0, Fr[Nf];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              nv[d] = CURVED ? nr[r][d] + nfv[d] : nfv[d];
              ub[d] = ah[r][d] + B.h[d];
              un = d ? fma(ub[d], nv[d], un) : ub[d] * nv[d];
              hv = d ? fma(2.0 * ah[r][d], B.h[d], hv) : 2.0 * ah[r][d] * B.h[d];
            }
            Fr[0] = rl[r] * un;
            Fr[DIM + 1] = fma(rl[r], fma(ib[r], pf[r], hv), pa[r]) * un;
            a0[r] = fma(w.x, Fr[0], a0[r]);
            aE[r] = fma(w.x, Fr[DIM + 1], aE[r]);
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              Fr[1 + d] = fma(Fr[0], ub[d], pa[r] * nv[d]);
              am[r][d] = fma(w.x, Fr[1 + d], am[r][d]);
            }
#pragma unroll
            for (int q = 0; q < Nf; ++q) af[q] = r ? fma(w.y, Fr[q], af[q]) : w.y * Fr[q];
          }
          if (on) {
#pragma unroll
            for (int q = 0; q < Nf; ++q) acc_f[q * NF + f] += af[q];
          }
        }
        __syncwarp();
      }
      if (SPLIT) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int d = 0; d < DIM; ++d) ap[r][d] = fma(pb[r], nb[d], ap[r][d]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      F[r][0] = a0[r];
      F[r][DIM + 1] = aE[r];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        F[r][1 + d] = am[r][d];
        if (SPLIT) {
          F[r][1 + d] = fma(ah[r][d], a0[r], am[r][d] + ap[r][d]);
          F[r][DIM + 1] = fma(2.0 * ah[r][d], am[r][d], F[r][DIM + 1]);
        }
      }
    }
  }

  // curved: n_i = sum_a nr_a G^a_i / 2 of the lane's rows for one face
  __device__ __forceinline__ void row_normals(const double *st, const int (&ir)[R], int fc,
                                              double (&nr)[R][DIM]) const {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        nr[r][d] = 0.0;
#pragma unroll
        for (int a = 0; a < DIM; ++a)
          nr[r][d] = fma(st[C::oG + (a * DIM + d) * Nq + ir[r]], sNr[fc * DIM + a], nr[r][d]);
      }
  }

  // the face row f of element ee that the pair phase has summed
  __device__ __forceinline__ void face_row(int ee, int f, double (&v)[Nf]) const {
    const double *acc_f = sAcc + ee * SA;
    if (!SPLIT) {
#pragma unroll
      for (int q = 0; q < Nf; ++q) v[q] = acc_f[q * NF + f];
      return;
    }
    const double *st = sSt + ee * SE, *nb = sNrm + ee * SN + f / Nfq * DIM;
    const double2 *q = (const double2 *)acc_f + f;
    const double2 q0 = q[0], q1 = q[NF], hb = ((const double2 *)(st + C::oB))[Nq + f];
    double m[DIM], hf[DIM], gE;
    m[0] = q1.x;
    m[1] = q1.y;
    hf[0] = hb.x;
    hf[1] = hb.y;
    if (DIM == 3) {
      const double2 q2 = q[2 * NF];
      m[DIM - 1] = q2.x;
      gE = q2.y;
      hf[DIM - 1] = st[C::oC + 2 * (Nq + f)];
    } else {
      gE = acc_f[4 * NF + f];
    }
    v[0] = q0.x;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      v[1 + d] = fma(hf[d], q0.x, fma(nb[d], q0.y, m[d]));
      gE = fma(2.0 * hf[d], m[d], gE);
    }
    v[DIM + 1] = gE;
  }

  // a face row back into its slots, for the lift (twice the row: the lift's
  // weights 1/2 VqLq are the pair phase's)
  __device__ __forceinline__ void put_row(int ee, int f, const double (&v)[Nf]) const {
    double *acc_f = sAcc + ee * SA;
    if (SPLIT) {
      double2 *q = (double2 *)acc_f + f;
      q[0].x = v[0];
      q[NF] = make_double2(v[1], v[2]);
      if (DIM == 3)
        q[2 * NF] = make_double2(v[3], v[Nf - 1]);
      else
        acc_f[4 * NF + f] = v[Nf - 1];
    } else {
#pragma unroll
      for (int q = 0; q < Nf; ++q) acc_f[q * NF + f] = v[q];
    }
  }
  __device__ __forceinline__ void get_row(const double *acc_f, int f, double (&v)[Nf]) const {
    if (SPLIT) {
      const double2 *q = (const double2 *)acc_f + f;
      v[0] = q[0].x;
      const double2 q1 = q[NF];
      v[1] = q1.x;
      v[2] = q1.y;
      if (DIM == 3) {
        const double2 q2 = q[2 * NF];
        v[3] = q2.x;
        v[Nf - 1] = q2.y;
      } else {
        v[Nf - 1] = acc_f[4 * NF + f];
      }
    } else {
#pragma unroll
      for (int q = 0; q < Nf; ++q) v[q] = acc_f[q * NF + f];
    }
  }

  // surface flux + Lax-Friedrichs penalty at the face points of the group's
  // batch elements [e0, e0 + G) (the TS threads t0, t0 + TS, ... of the
  // group), added to the face rows: sf = rhsQf + 1/2
  // F_S(u-, u+).nJ - tau/4 max(lam-, lam+) sJ (u+ - u-) (Euler3D.okl:3256-3346,
  // Euler2D.okl:1373-1453).  The plus trace is gathered
  // from uf through mapPq (the neighbour indices of all of a thread's face
  // points are loaded first).
  template <int TS>
  __device__ __forceinline__ void surface(int K, int k0, int e0, int t0,
                                          const double *__restrict__ fgeo,
                                          const uint32_t *__restrict__ mapPq, const double *uf,
                                          const Phys &P) const {
    constexpr int NFG = El::Nfgeo, NPT = (G * NF + TS - 1) / TS;
    // point u of the thread: its element (in the group) and face node; those
    // past the group's or the mesh's end repeat a valid one and are not stored
    auto el = [&](int u) { return min(min((t0 + u * TS) / NF, G - 1), K - 1 - k0 - e0); };
    uint32_t idP[NPT];
#pragma unroll
    for (int u = 0; u < NPT; ++u)
      idP[u] = mapPq[(t0 + u * TS) % NF + (size_t)(k0 + e0 + el(u)) * NF];
    struct Point {
      double nJ[DIM], sJ, UM[Nf], UP[Nf];
    };
    auto fetch = [&](int u) {
      Point p;
      const int f = (t0 + u * TS) % NF;
      const size_t k = k0 + e0 + el(u);
      const double *fg = fgeo + k * NF * NFG + f, *um = uf + k * NF * Nf + f, *up = uf + idP[u];
#pragma unroll
      for (int d = 0; d < DIM; ++d) p.nJ[d] = fg[d * NF];
      p.sJ = fg[DIM * NF];
#pragma unroll
      for (int q = 0; q < Nf; ++q) {
        p.UM[q] = um[q * NF];
        p.UP[q] = up[q * NF];
      }
      return p;
    };
    Point p = fetch(0);
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
      Point next;
      if (u + 1 < NPT) next = fetch(u + 1);  // in flight during this point's arithmetic
      const int t = t0 + u * TS, ee = e0 + t / NF, f = t % NF;
      double kM, kP, c2M, c2P;
      const NodeState<DIM> M = node_state_surf<DIM>(p.UM, 1, P, kM, c2M);
      const NodeState<DIM> Pp = node_state_surf<DIM>(p.UP, 1, P, kP, c2P);
      double F[Nf], v[Nf];
      ecflux_n_nolog<DIM, true>(M, Pp, p.nJ, P, F);
      const double lamM = fsqrt(kM) + fsqrt(c2M);
      const double lamP = fsqrt(kP) + fsqrt(c2P);
      const double tau = (DIM == 3) ? P.tau : 1.0;
      const double Lfc = tau * 0.25 * fmax(lamM, lamP) * p.sJ;
      if (t < G * NF && k0 + ee < K) {
        face_row(ee, f, v);
#pragma unroll
        for (int q = 0; q < Nf; ++q) v[q] = fma(-2.0 * Lfc, p.UP[q] - p.UM[q], fma(2.0, v[q], F[q]));
        put_row(ee, f, v);
      }
      if (u + 1 < NPT) p = next;
    }
  }

  // lift: rows += (1/2 VqLq) (2 sf) on the rotated weights, the warps of
  // the group splitting the face nodes as in the pair phase
  __device__ __forceinline__ void lift(double (&acc)[R][Nf]) const {
    const double *sf = sAcc + e * SA;
#pragma unroll 1
    for (int fb = T::f0(h); fb < T::f0(h) + T::nf(h); fb += FACES ? Nfq : NF) {
      const int n = steps(h);
      const double *wb = sW + 2 * (weights(fb) + l);
      for (int s = 0; s < n; ++s) {
        const int ff = node(l, s, n);
        double v[Nf];
        get_row(sf, fb + (IDLE ? min(ff, Nfq - 1) : ff), v);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double w = wb[2 * (s * R + r) * L];
#pragma unroll
          for (int q = 0; q < Nf; ++q) acc[r][q] = fma(w, v[q], acc[r][q]);
        }
      }
    }
  }

  // the per-node logarithms of the batch elements [e0, e0 + ne) (threads t0,
  // t0 + ts, ...), from the stored density and beta
  __device__ __forceinline__ void fill_logs(int e0, int ne, int t0, int ts) const {
    for (int t = t0; t < ne * NN; t += ts) {
      double *st = sSt + (e0 + t / NN) * SE;
      const int n = t % NN;
      const double2 a = ((const double2 *)(st + C::oA))[n];
      ((double2 *)st)[n] = make_double2(log(2.0 * a.x), log(a.y));
    }
  }

  // The pair phase of the group (H warps, threads t0 .. t0 + ts - 1 over
  // the batch elements [e0, e0 + G), `gsync` its barrier): the pair loops of
  // the range that the group's states span; the logarithms only where the
  // log-difference may be needed.
  template <typename Sync>
  __device__ __forceinline__ void group_pairs(double (&acc)[R][Nf], const Phys &P, int e0, int t0,
                                              int ts, Sync gsync) const {
    const double *st = sSt + e * SE;
    const int range = state_range<NN, L>(l, [&](int n, int &r, int &b) {
      const double2 a = ((const double2 *)(st + C::oA))[n];
      r = __double2hiint(a.x);
      b = __double2hiint(a.y);
    });
    if (range == 0) {
      pairs<0>(acc, P);
    } else if (range == 1) {
      pairs<1>(acc, P);
    } else if (range == 2) {
      pairs<2>(acc, P);
    } else {
      fill_logs(e0, G, t0, ts);
      gsync();
      pairs<3>(acc, P);
    }
  }

  // the warps but the first park their partial rows in element e's state block
  // ([H - 1][Nf][Nq]; the group's pairs are done).  With two warps they lie over the
  // logarithms and densities, which face_row does not read; else the face rows
  // must have been read too
  __device__ __forceinline__ void park_rows(const double (&acc)[R][Nf]) const {
    static_assert(Nf * Nq <= 4 * NN && (H - 1) * Nf * Nq <= SE, "row buffer");
    double *rowbuf = sSt + e * SE + (h - 1) * Nf * Nq;
    if (h >= 1) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = l + L * r;
        if (i < Nq) {
#pragma unroll
          for (int q = 0; q < Nf; ++q) rowbuf[q * Nq + i] = acc[r][q];
        }
      }
    }
  }
  // field q of row i, summed over the group's warps (the first warp's sum in a)
  __device__ __forceinline__ double row_sum(double a, int q, int i) const {
    const double *rowbuf = sSt + e * SE + q * Nq + i;
#pragma unroll
    for (int hh = 1; hh < H; ++hh) a += rowbuf[(hh - 1) * Nf * Nq];
    return a;
  }
};

// SURF = false: the volume kernel (euler_vol_*): rhsQ <- the volume rows,
// rhsQf <- the face rows.  SURF = true: the volume and the surface kernel of
// a stage in one launch: after the pairs, the group adds the surface flux and
// penalty to its face rows (gathering the neighbours' traces from Qf through
// mapPq; Qf is only read, so every element's traces are final) and lifts
// them into its rows; rhsQ <- the whole right-hand side the surface kernel
// would leave, rhsQf is not written (fgeo and mapPq unused when false)
template <int DIM, int N, bool CURVED, int W, bool SURF = false, int RR = 0, int HH = 0>
__global__ void __launch_bounds__(HH ? 384 : 32 * W, 1)  // (with a warp per face: 168 registers at any W)
vol_pairs_kernel(int K, const double *__restrict__ vgeo, const double *__restrict__ vfgeo,
                 const double *__restrict__ nrJ, const double *__restrict__ nsJ,
                 const double *__restrict__ ntJ, const double *__restrict__ Drq,
                 const double *__restrict__ Dsq, const double *__restrict__ Dtq,
                 const double *__restrict__ VqLq, const double *__restrict__ VfPq,
                 const double *Qf, double *rhsQ, double *rhsQf, Phys P,
                 const double *__restrict__ fgeo = nullptr,
                 const uint32_t *__restrict__ mapPq = nullptr,
                 const int *__restrict__ blist = nullptr, const int *__restrict__ nblist = nullptr) {
  using V = VolPairs<DIM, N, CURVED, W, RR, HH>;
  constexpr int Nq = V::Nq, NF = V::NF, Nf = V::Nf, R = V::R, L = V::L, E = V::C::EB, H = V::H;
  extern __shared__ double smem[];
  V v(smem);
  constexpr bool PRE = V::C::PREFETCH;
  // After the tables, the H warps of an element group touch only their own
  // G elements' shared memory (states, face rows, normals, staged traces),
  // so within the batch loop they synchronise among themselves (a named
  // barrier per group) and never wait for the CTA's other groups.
  constexpr int G = V::G, GT = 32 * H;
  const int q = (threadIdx.x >> 5) / H, tq = threadIdx.x - q * GT;
  auto gsync = [&] {
    if (H == 1)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;\n" ::"r"(1 + q), "r"(GT) : "memory");
  };
  // stage the group's elements from kq on (face traces, a contiguous range
  // of Qf) into shared memory
  // (without room for them: into L2), and the affine elements' geometric factors
  auto prefetch_group = [&](int kq) {
    if (kq < K) {
      const int n = min(K - kq, G) * NF * Nf;
      const double *src = Qf + (size_t)kq * NF * Nf;
      if (PRE) {
        double *dst = v.sPre + (size_t)q * G * NF * Nf;
        for (int t = tq; t < n; t += GT) cp_async8(dst + t, src + t);
      } else {
        prefetch_lines(src, n * 8, tq, GT);
      }
      v.fetch_geo(K, kq - q * G, q * G, tq, GT, vgeo);
      prefetch_lines(rhsQ + (size_t)kq * Nq * Nf, min(K - kq, G) * Nq * Nf * 8, tq, GT);
      if (CURVED) {
        prefetch_lines(vgeo + (size_t)kq * Nq * V::NG, min(K - kq, G) * Nq * V::NG * 8, tq, GT);
        prefetch_lines(vfgeo + (size_t)kq * NF * V::NG, min(K - kq, G) * NF * V::NG * 8, tq, GT);
      }
      if (SURF) {
        prefetch_lines(fgeo + (size_t)kq * NF * V::El::Nfgeo, min(K - kq, G) * NF * V::El::Nfgeo * 8, tq, GT);
        prefetch_lines(mapPq + (size_t)kq * NF, min(K - kq, G) * NF * 4, tq, GT);
      }
    }
    cp_async_commit();
  };
  // The work: batches of E elements, all of them or (a work list: the
  // ensemble's active instances) the ascending batch indices blist[0 ..
  // *nblist), each cut into its NG group slices of G elements.  The groups
  // take the slices independently: in round i group q of CTA b (of W / H) takes
  // slice (i W / H + q) grid + b, so a last, partial round leaves the busy groups
  // spread over every SM (rather than whole CTAs busy and the other SMs
  // idle).  Every slice is G consecutive elements, so the elements that
  // share a warp, and the results, do not depend on the schedule.
  constexpr int NG = E / G;
  const int nb = blist ? *nblist : (K + E - 1) / E;
  const int ns = nb * NG, sstep = (int)gridDim.x * (W / H);
  auto slice = [&](int g) {  // first element of slice g (K past the end)
    if (g >= ns) return K;
    const int cb = g / NG;
    return (blist ? blist[cb] : cb) * E + (g - cb * NG) * G;
  };
  const int g0 = q * (int)gridDim.x + (int)blockIdx.x;
  if (HH > 0) {  // launched to overlap the previous kernel's end on the smallest meshes
    pdl_trigger();
    v.load_tables(nrJ, nsJ, ntJ, Drq, Dsq, Dtq, VqLq, VfPq);  // no kernel's output
    pdl_wait();
    prefetch_group(slice(g0));
  } else {
    prefetch_group(slice(g0));
    v.load_tables(nrJ, nsJ, ntJ, Drq, Dsq, Dtq, VqLq, VfPq);
  }
  __syncthreads();  // the tables are shared by every group

  for (int gi = g0; gi < ns; gi += sstep) {
    const int kg = slice(gi);
    cp_async_wait_all();
    // a slice whose elements all lie past the end (of a partial last batch)
    // has nothing to compute, and must not read element K-1's input, which
    // the group owning it may already have overwritten with its RHS
    if (kg >= K) break;
    // the helpers index the group's elements as k0 + q G + (0 .. G-1)
    const int k0 = kg - q * G;
    gsync();  // the group's traces staged / its previous slice done with its shared memory
    v.template prologue_group<GT>(K, k0, q * G, tq, vgeo, vfgeo, rhsQ, Qf, P, PRE ? v.sPre : nullptr);
    gsync();
    prefetch_group(slice(gi + sstep));  // the next slice's traces, during the pairs
    double acc[R][Nf];
    v.group_pairs(acc, P, q * G, tq, GT, gsync);
    gsync();  // the group's pairs done
    if (SURF) {
      v.template surface<GT>(K, k0, q * G, tq, fgeo, mapPq, Qf, P);
      gsync();  // face rows complete: lift
      v.lift(acc);
    } else {
      for (int t = tq; t < G * NF; t += GT) {
        const int ee = q * G + t / NF, f = t % NF;
        if (k0 + ee >= K) continue;
        double row[Nf];
        v.face_row(ee, f, row);
        double *outf = rhsQf + (size_t)(k0 + ee) * NF * Nf + f;
#pragma unroll
        for (int c = 0; c < Nf; ++c) outf[c * NF] = row[c];
      }
    }
    if (!SURF && H > 2) gsync();  // face rows read: the states become the row buffers
    v.park_rows(acc);
    gsync();
    const int k = k0 + v.e;
    if (k < K && v.h == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = v.l + L * r;
        if (i < Nq) {
          double *out = rhsQ + (size_t)k * Nq * Nf + i;
#pragma unroll
          for (int q = 0; q < Nf; ++q) out[q * Nq] = v.row_sum(acc[r][q], q, i);
        }
      }
    }
  }
}

}  // namespace wadg
