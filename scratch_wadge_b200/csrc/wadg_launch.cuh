// Launches of the volume, surface, update and fused stage kernels: CTA shapes,
// grids and the choice among them.  The function templates are instantiated
// once per (dim, N) in wadg_k<dim><N>.cu, so that the degrees compile in
// parallel; wadg_capi.cu calls them.
#pragma once

#include <cuda_runtime.h>

#include "../../include/wadg.h"
#include "wadg_host.h"
#include "wadg_stage.cuh"
#include "wadg_surf_mma.cuh"
#include "wadg_update_mma.cuh"
#include "wadg_vol.cuh"

struct wadg_ctx {
  int dim, N, Nq, Nfq, Nfaces;
  wadg::Phys phys;
  cudaStream_t stream;
  int vol_warps = 0;  // warps per CTA of the pair volume kernel; 0 = the default
  int vol_rows = 0;   // rows per lane of its node-to-thread map; 0 = the default
  bool overlap = false;  // kernels may overlap their predecessor's end (overlaps())
};

namespace wadg {

int fail(int code, const char *fmt, ...);  // wadg_capi.cu: sets wadg_last_error, returns code
int cuda_check(cudaError_t e, const char *what);

inline int after_launch(const char *name) { return cuda_check(cudaGetLastError(), name); }

// warps per CTA of the pair-scheduled volume kernel: as many as fit in 227 KB
// of shared memory, at most `cap`; from 8 on a multiple of 4, the same number on
// each quarter of the SM (10 warps leave 3 on two of them and 168 registers per
// thread as with 12, so they run as long as 12 would for 10/12 of the work: curved
// 3D N=4, K=10368 0.40 ms with 10 warps, 0.33 with 8)
template <int DIM, int N, bool CURVED, int RR = 0>
constexpr int volpairsW_fit(int cap) {
  using C = VolPairsCfg<DIM, N, CURVED, 2, RR>;
  constexpr size_t per_warp = C::per_elem * VolTile<DIM, N, RR>::G / C::H;
  constexpr size_t w = (227 * 1024 - C::fixed) / per_warp;
  return w >= (size_t)cap ? cap : (w < 2 ? 2 : (int)(w < 8 ? w & ~size_t(1) : w & ~size_t(3)));
}

// the default shape: at most 12 warps (register budget ~170 per thread)
template <int DIM, int N, bool CURVED>
constexpr int volpairsW() {
  return volpairsW_fit<DIM, N, CURVED>(12);
}

inline int num_sms() { return wadg_internal::sm_count(); }

// Whether a kernel over K elements may start before its predecessor has
// finished (programmatic dependent launch; the kernel reads nothing that a
// predecessor writes before its griddepcontrol.wait).  Only while the app
// captures a time step of its own kernels (c->overlap), and only on meshes with
// at most one element group per SM, where launch and table loads are a good
// part of a kernel: 10 time steps of 162 tets N=2 0.753 -> 0.690 ms, 200
// triangles N=2 0.644 -> 0.636 ms; no gain at 1.7 groups per SM (2048 triangles
// N=3), and Taylor-Green K=24576 1.38 -> 1.45 ms per step
template <int DIM, int N>
bool overlaps(const wadg_ctx *c, int K) {
  return c->overlap && K <= VolTile<DIM, N>::G * num_sms();
}

// a kernel on the context's stream.  The error of a failed launch is taken off the
// runtime's record: left there, it would be the next call's
template <class... KA, class... A>
int launch(const wadg_ctx *c, const char *name, bool overlap, void (*kern)(KA...), int grid, int threads,
           size_t smem, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, KA(args)...);
  return after_launch(name);
}

// CTAs of a persistent kernel over K elements in batches of E: one per batch,
// at most as many as are resident at once (shared memory per CTA `smem`); CTA
// b takes batches b, b + grid, b + 2 grid, ...
inline int persistent_grid(int K, int E, size_t smem) {
  const int per_sm = (int)((227 * 1024) / smem) > 0 ? (int)((227 * 1024) / smem) : 1;
  const int batches = (K + E - 1) / E;
  return batches < num_sms() * per_sm ? batches : num_sms() * per_sm;
}

// CTAs of the volume kernel: its element groups take slices of G elements, slice
// s going to CTA s mod grid first, so one CTA per slice up to one per SM, and
// more per SM only when the slices outnumber those CTAs' groups: a mesh of few
// slices runs one group on each of many SMs rather than all of a CTA's groups on
// few (10 time steps, one CTA per batch before: 162 tets N=2 1.39 -> 1.03 ms,
// 2146 curved triangles N=4 1.57 -> 1.42 ms, 2048 triangles N=3 1.01 -> 0.94 ms)
template <class C>
int vol_grid(int K) {
  const int slices = (K + C::T::G - 1) / C::T::G, groups = C::threads / 32 / C::H;
  if (slices <= num_sms() * groups) return slices < num_sms() ? slices : num_sms();
  return persistent_grid(K, C::T::G, C::smem_vol);
}

// candidate CTA shapes of the pair volume kernel (warps per CTA; elements per
// CTA = warps / 2 * 32 / lanes per element): the default, then two and four
// warps fewer.  In 2D the second is 16 warps where they fit: four fields need
// fewer registers (128 per thread).  Which count is fastest goes with the rounds
// that a mesh's slices make of it (default_warps)
template <int DIM, int N, bool CURVED>
constexpr int volpairsW_cand(int i) {
  constexpr int W0 = volpairsW<DIM, N, CURVED>();
  constexpr int Wbig = DIM == 2 ? volpairsW_fit<DIM, N, CURVED>(16) : W0;
  if (i == 1 && Wbig > W0) return Wbig;
  return i == 0 ? W0 : (W0 - 2 * i >= 2 ? W0 - 2 * i : 0);
}

// More counts of warps that wadg_ctx_set_vol_warps takes, though they are no candidates:
// they were, while an element took more shared memory
template <int DIM, int N, bool CURVED>
constexpr int volpairsW_more(int i) {
  if (DIM == 3 && CURVED && N <= 2) return i == 0 ? 6 : N == 2 ? 4 : 0;
  return DIM == 2 && N == 1 && !CURVED && i == 0 ? 10 : 0;
}

// The other node-to-thread maps: half and twice the default's lanes per
// element (about twice and half its rows per lane), each given to the kernels
// as RR = rows per lane.  A map is a candidate when it has as many lanes as
// intended (2 to 32), keeps a face node per lane in each warp's face half,
// pads no more node slots than the default, holds at most 4 rows per lane and
// fits a CTA of at least 4 warps in shared memory.  (Six rows per lane need
// more than 255 registers in 3D: 140-530 bytes of spills at every degree.)
// alt_rows<DIM, N, CURVED, j>(), j = 0 (half the lanes) or 1 (twice): its RR,
// or 0 when it is no candidate; its warps per CTA: the most that fit, up to 16
// with at most two rows per lane, else 8 (up to 255 registers per thread).
template <int DIM, int N, int RR>
struct NodeMap {  // VolTile's arithmetic, without its static checks
  static constexpr int Nq = Elem<DIM, N>::Nq;
  static constexpr int Lraw = RR > 0 ? (Nq + RR - 1) / RR : (Nq + 2) / 3;
  static constexpr int L = Lraw <= 1 ? 1 : Lraw <= 2 ? 2 : Lraw <= 4 ? 4 : Lraw <= 8 ? 8 : Lraw <= 16 ? 16 : 32;
  static constexpr int R = (Nq + L - 1) / L;
  static constexpr int pad = L * R - Nq;
};
template <int DIM, int N, bool CURVED, int RR>
constexpr int alt_warps() {
  return volpairsW_fit<DIM, N, CURVED, RR>(NodeMap<DIM, N, RR>::R <= 2 ? 16 : 8);
}
template <int DIM, int N, bool CURVED, int j>
constexpr int alt_rows() {
  constexpr int L0 = NodeMap<DIM, N, 0>::L, Lt = j == 0 ? L0 / 2 : 2 * L0;
  if constexpr (Lt < 2 || Lt > 32) {
    return 0;
  } else {
    constexpr int RR = (Elem<DIM, N>::Nq + Lt - 1) / Lt;
    using M = NodeMap<DIM, N, RR>;
    // (nf1: the smaller face half, the second warp's when there are two)
    constexpr int nf1 = Elem<DIM, N>::NfqNf / 2;
    constexpr int faces = nf1 >= M::L ? nf1 : Elem<DIM, N>::NfqNf;
    if constexpr (M::L != Lt || faces < M::L || M::pad > NodeMap<DIM, N, 0>::pad || M::R > 4) {
      return 0;
    } else {
      constexpr int W = alt_warps<DIM, N, CURVED, RR>();
      return (W >= 4 && VolPairsCfg<DIM, N, CURVED, W, RR>::smem <= 227 * 1024) ? RR : 0;
    }
  }
}

// Small meshes take a warp per face (HH = Nfaces, 12 warps) instead of two (or
// one) per element group: a slice then has half as many pair steps one after another,
// which is what bounds a kernel of a slice or two per group; fewer groups fit an SM
// (3 for 6 in 3D, 4 for 6 or 12 in 2D).  So: while the slices are at most
// one per such group of an SM.  Volume + surface kernel, ms without -> with, by
// slices per SM: 2D N=3 1.7 .0158 -> .0123, 3.9 .0158 -> .0124, K=32768 (28)
// .0496 -> .0572; 3D N=2 0.1 .0125 -> .0084, 2.6 .0165 -> .0132, 21 .0745 -> .0777;
// N=3 0.6 .0162 -> .0111, 2.2 .0222 -> .0186, 5.2 .0312 -> .0339, 42 .200 -> .222;
// curved N=3 2.2 .0354 -> .0287, 3.5 .0328 -> .0391; curved N=4 2.5 .0528 -> .0401;
// 2D curved N=4 (faces of 5 nodes, 8 lanes: 3 idle) 3.6 .0244 -> .0166, 14 .0299 -> .0415
template <int DIM, int N, bool CURVED>
constexpr int faces_warps() {
  return VolTile<DIM, N>::H < Elem<DIM, N>::Nfaces ? Elem<DIM, N>::Nfaces : 0;
}
template <int DIM, int N>
int slices_per_sm(int K) {
  const int slices = (K + VolTile<DIM, N>::G - 1) / VolTile<DIM, N>::G;
  return (slices + num_sms() - 1) / num_sms();
}
template <int DIM, int N, bool CURVED>
bool small_mesh(const wadg_ctx *c, int K) {
  if (faces_warps<DIM, N, CURVED>() == 0 || c->vol_warps || c->vol_rows) return false;
  return slices_per_sm<DIM, N>(K) <= 12 / Elem<DIM, N>::Nfaces;
}

// Warps per CTA of the default map: the context's choice, else the default (0), or 16
// in 2D where they finish in a round fewer (at most two, as their 128
// registers per thread cost 2 % in longer runs).  10 time steps, ms, 12 -> 16
// warps, by slices per SM: N=3 (6 groups for 8) 6.9 1.318 -> 1.223, 13.8 2.10 ->
// 2.02; curved N=3 6.9 1.58 -> 1.44; N=2 13.8 2.31 -> 2.17; curved N=2 6.9 1.70 ->
// 1.53; curved N=4 (12 groups for 16) 12.2 2.05 -> 1.83.  Volume + surface kernel alone
// at N=4, 16 warps' time over 12's by slices per SM: curved 13.0-13.8 1.00-1.02, 15.6
// 0.91, 25.9-31.6 0.84-1.03; affine (not taken) 12.3 0.93, 13.0-13.8 1.00-1.01, 15.6 0.92,
// 26-31 1.02-1.05; volume + surface kernel, us, N=1 6.5 23.8 -> 19.6, 7.4 24.3 -> 21.4,
// 13.0 33.7 -> 30.2.  Curved 3D N=2: eight where twelve save no round (255 registers a
// thread for 168), us, 12 -> 8 warps, smooth / random states: 3.7 29.5 -> 27.5 / 40.5 ->
// 38.9; 6.7 48.7 -> 43.9 / 70.0 -> 65.3; 5.1 (a round against two) 34.6, 8 warps 39.1.  Same bits
template <int DIM, int N, bool CURVED>
int default_warps(const wadg_ctx *c, int K) {
  constexpr int W0 = volpairsW<DIM, N, CURVED>(), W1 = volpairsW_cand<DIM, N, CURVED>(1);
  if (DIM == 3 && CURVED && N == 2 && !c->vol_warps && !c->vol_rows) {
    const int m = slices_per_sm<DIM, N>(K), g = W0 / VolTile<DIM, N>::H, g8 = 8 / VolTile<DIM, N>::H;
    return (m + g8 - 1) / g8 <= (m + g - 1) / g ? 8 : 0;
  }
  if (c->vol_warps || c->vol_rows || DIM == 3 || (N == 4 && !CURVED) || W1 <= W0) return c->vol_warps;
  constexpr int g0 = W0 / VolTile<DIM, N>::H, g1 = W1 / VolTile<DIM, N>::H;
  const int m = slices_per_sm<DIM, N>(K);
  return m <= 2 * g1 && (m + g1 - 1) / g1 < (m + g0 - 1) / g0 ? W1 : 0;
}

// The CTA of a small mesh: with two slices per SM the warps of two, so that other
// streams' CTAs fit beside it (three or four slices take all 12; with one, a CTA of its
// own warps alone loads the tables 0.5-1 us slower and, launched ahead, stacks on few SMs:
// 750 tets N=2 0.60 -> 0.73 ms for 10 time steps).  Solves of 2048 triangles N=3 on
// streams of their own, us per time step of all, 12 warps -> 6: one 82 -> 82, two 111 ->
// 95, four 161 -> 125, eight 318 -> 221; 1296 tets N=2, 12 -> 8: one 90 -> 90, four 187 -> 162
template <int W_, int RR_ = 0, int HH_ = 0>
struct VolShape {
  static constexpr int W = W_, RR = RR_, HH = HH_;
};

// f(VolShape) with the shape of the volume kernels for K elements: the context's
// (wadg_ctx_set_vol_shape), else the automatic one
template <int DIM, int N, bool CURVED, class F>
int with_vol_shape(const wadg_ctx *c, int K, F f) {
  constexpr int HH = faces_warps<DIM, N, CURVED>();
  if constexpr (HH > 0)
    if (small_mesh<DIM, N, CURVED>(c, K))
      return slices_per_sm<DIM, N>(K) == 2 ? f(VolShape<2 * HH, 0, HH>()) : f(VolShape<12, 0, HH>());
  constexpr int A0 = alt_rows<DIM, N, CURVED, 0>(), A1 = alt_rows<DIM, N, CURVED, 1>();
  if constexpr (A0 > 0)
    if (c->vol_rows == A0) return f(VolShape<alt_warps<DIM, N, CURVED, A0>(), A0>());
  if constexpr (A1 > 0)
    if (c->vol_rows == A1) return f(VolShape<alt_warps<DIM, N, CURVED, A1>(), A1>());
  constexpr int W0 = volpairsW<DIM, N, CURVED>();
  constexpr int W1 = volpairsW_cand<DIM, N, CURVED>(1), W2 = volpairsW_cand<DIM, N, CURVED>(2);
  constexpr int W3 = volpairsW_more<DIM, N, CURVED>(0), W4 = volpairsW_more<DIM, N, CURVED>(1);
  const int warps = default_warps<DIM, N, CURVED>(c, K);
  if (W1 && warps == W1) return f(VolShape<(W1 ? W1 : W0)>());
  if (W2 && warps == W2) return f(VolShape<(W2 ? W2 : W0)>());
  if (W3 && warps == W3) return f(VolShape<(W3 ? W3 : W0)>());
  if (W4 && warps == W4) return f(VolShape<(W4 ? W4 : W0)>());
  return f(VolShape<W0>());
}

// SURF: the volume + surface kernel (rhsQf unused; fgeo, mapPq read)
template <int DIM, int N, bool CURVED, int W, bool SURF = false, int RR = 0, int HH = 0>
int launch_vol_pairs_w(const wadg_ctx *c, int K, const double *vgeo, const double *vfgeo,
                       const double *nrJ, const double *nsJ, const double *ntJ, const double *Drq,
                       const double *Dsq, const double *Dtq, const double *VqLq, const double *VfPq,
                       const double *Qf, double *rhsQ, double *rhsQf,
                       const double *fgeo = nullptr, const uint32_t *mapPq = nullptr,
                       const int *blist = nullptr, const int *nb = nullptr) {
  using C = VolPairsCfg<DIM, N, CURVED, W, RR, HH>;
  static_assert(C::smem_vol <= 227 * 1024, "pair-scheduled volume kernel does not fit in shared memory");
  auto kern = vol_pairs_kernel<DIM, N, CURVED, W, SURF, RR, HH>;
  static wadg_internal::PerDevice<bool> attr;
  if (!attr.here()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem_vol);
    if (e != cudaSuccess) return cuda_check(e, "volume kernel smem attribute");
    attr.here() = true;
  }
  const int grid = vol_grid<C>(K);
  return launch(c, SURF ? "volume + surface kernel" : "volume kernel", HH > 0 && overlaps<DIM, N>(c, K),
                kern, grid, C::threads, C::smem_vol, K, vgeo, vfgeo, nrJ, nsJ, ntJ, Drq, Dsq, Dtq, VqLq, VfPq,
                Qf, rhsQ, rhsQf, c->phys, fgeo, mapPq, blist, nb);
}

template <int DIM, int N, bool CURVED>
int launch_volsurf(const wadg_ctx *c, int K, const double *vgeo, const double *vfgeo,
                   const double *fgeo, const uint32_t *mapPq, const double *nrJ,
                   const double *nsJ, const double *ntJ, const double *Drq, const double *Dsq,
                   const double *Dtq, const double *VqLq, const double *VfPq, const double *Qf,
                   double *rhsQ, const int *blist = nullptr, const int *nb = nullptr) {
  return with_vol_shape<DIM, N, CURVED>(c, K, [&](auto s) {
    using S = decltype(s);
    return launch_vol_pairs_w<DIM, N, CURVED, S::W, true, S::RR, S::HH>(
        c, K, vgeo, vfgeo, nrJ, nsJ, ntJ, Drq, Dsq, Dtq, VqLq, VfPq, Qf, rhsQ, nullptr, fgeo, mapPq, blist, nb);
  });
}

template <int DIM, int N, bool CURVED>
int launch_vol_pairs(const wadg_ctx *c, int K, const double *vgeo, const double *vfgeo,
                     const double *nrJ, const double *nsJ, const double *ntJ, const double *Drq,
                     const double *Dsq, const double *Dtq, const double *VqLq, const double *VfPq,
                     const double *Qf, double *rhsQ, double *rhsQf) {
  return with_vol_shape<DIM, N, CURVED>(c, K, [&](auto s) {
    using S = decltype(s);
    return launch_vol_pairs_w<DIM, N, CURVED, S::W, false, S::RR, S::HH>(
        c, K, vgeo, vfgeo, nrJ, nsJ, ntJ, Drq, Dsq, Dtq, VqLq, VfPq, Qf, rhsQ, rhsQf);
  });
}

template <int DIM, int N, bool CURVED>
int vol_warps_more(int *out) {
  int n = 0;
  for (int i = 0; i < 2; ++i)
    if (int w = volpairsW_more<DIM, N, CURVED>(i)) out[n++] = w;
  return n;
}

template <int DIM, int N, bool CURVED>
int vol_warps_candidates(int *out) {
  int n = 0;
  for (int i = 0; i < 3; ++i)
    if (int w = volpairsW_cand<DIM, N, CURVED>(i)) out[n++] = w;
  return n;
}

// every compiled (warps, rows) shape: the default map's warps, then the
// other maps (rows > 0)
template <int DIM, int N, bool CURVED>
int vol_shapes(int *warps, int *rows) {
  int n = vol_warps_candidates<DIM, N, CURVED>(warps);
  for (int i = 0; i < n; ++i) rows[i] = 0;
  constexpr int A0 = alt_rows<DIM, N, CURVED, 0>(), A1 = alt_rows<DIM, N, CURVED, 1>();
  if constexpr (A0 > 0) {
    warps[n] = alt_warps<DIM, N, CURVED, A0>();
    rows[n++] = A0;
  }
  if constexpr (A1 > 0) {
    warps[n] = alt_warps<DIM, N, CURVED, A1>();
    rows[n++] = A1;
  }
  return n;
}

// f(warps per CTA) of the fused stage kernel for K elements: the volume kernel's default,
// but at curved 3D N=2 eight where twelve save no round (255 registers a thread for 168, and
// the stage spills 80 bytes at 168).  us, 12 -> 8 warps: K=162 36.9 -> 27.7, 7986 (two
// rounds either way) 68.2 -> 51.5; 24576 (four rounds, or six) 156 at 12
template <int DIM, int N, bool CURVED, class F>
int with_stage_warps(int K, F f) {
  constexpr int W = stage_warps<DIM, N, CURVED, volpairsW<DIM, N, CURVED>()>();
  if constexpr (DIM == 3 && CURVED && N == 2) {
    constexpr int E = VolPairsCfg<DIM, N, CURVED, W>::E, E8 = VolPairsCfg<DIM, N, CURVED, 8>::E;
    auto rounds = [&](int e) { return ((K + e - 1) / e + num_sms() - 1) / num_sms(); };
    if (rounds(E8) <= rounds(E)) return f(IntTag<8>());
  }
  return f(IntTag<W>());
}

template <int DIM, int N, bool CURVED>
int launch_stage(const wadg_ctx *c, int K, const double *vgeo, const double *vfgeo,
                 const double *fgeo, const uint32_t *mapPq, const double *nrJ, const double *nsJ,
                 const double *ntJ, const double *Drq, const double *Dsq, const double *Dtq,
                 const double *VqLq, const double *VfPq, const double *VqPq, const double *Jq,
                 double fa, double fb, double fdt, const double *uq, const double *uf, double *Q,
                 double *resQ, double *uq_out, double *uf_out) {
  if (uf_out == uf) return fail(WADG_ERR_INVALID, "stage: uf_out must not be uf");
  return with_stage_warps<DIM, N, CURVED>(K, [&](auto w) {
    constexpr int W = decltype(w)::value;
    using C = VolPairsCfg<DIM, N, CURVED, W>;
    auto kern = stage_kernel<DIM, N, CURVED, W>;
    static wadg_internal::PerDevice<bool> attr;
    if (!attr.here()) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem_vol);
      if (e != cudaSuccess) return cuda_check(e, "stage kernel smem attribute");
      attr.here() = true;
    }
    const int grid = persistent_grid(K, C::E, C::smem_vol);
    kern<<<grid, C::threads, C::smem_vol, c->stream>>>(K, vgeo, vfgeo, fgeo, mapPq, nrJ, nsJ, ntJ, Drq,
                                                    Dsq, Dtq, VqLq, VfPq, VqPq, Jq, fa, fb, fdt, uq,
                                                    uf, Q, resQ, uq_out, uf_out, c->phys);
    return after_launch("stage kernel");
  });
}

template <int DIM, int N>
int launch_surf(const wadg_ctx *c, int K, const double *fgeo, const uint32_t *mapPq,
                const double *VqLq, const double *Qf, const double *rhsQf, double *rhsQ) {
  using C = SurfMmaCfg<DIM, N>;
  return launch(c, "surf kernel", overlaps<DIM, N>(c, K), surf_mma_kernel<DIM, N>, (K + C::EW - 1) / C::EW,
                C::threads, C::smem, K, fgeo, mapPq, VqLq, Qf, rhsQf, rhsQ, c->phys);
}

// CTAs of the persistent update kernel: one per group of C::EW elements, at
// most as many as are resident at once (occupancy, cached per device)
template <int DIM, int N, bool CURVED>
int update_grid(int K, int *grid) {
  using C = UpdMmaCfg<DIM, N, CURVED>;
  auto kern = update_mma_kernel<DIM, N, CURVED>;
  static wadg_internal::PerDevice<int> per_sm_dev;
  int &per_sm = per_sm_dev.here();
  if (!per_sm) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem);
    if (e != cudaSuccess) return cuda_check(e, "update kernel smem attribute");
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, C::threads, C::smem);
    if (e != cudaSuccess) return cuda_check(e, "update kernel occupancy");
    per_sm = n < 1 ? 1 : n;
  }
  const int ctas = (K + C::EW - 1) / C::EW;
  *grid = ctas < num_sms() * per_sm ? ctas : num_sms() * per_sm;
  return WADG_OK;
}

// the launch shape of one kernel for K elements (wadg_kernel_shape)
template <int DIM, int N, bool CURVED>
int kernel_shape(const wadg_ctx *c, int kernel, int K, int *E, int *grid) {
  switch (kernel) {
    case WADG_KERNEL_VOL:
    case WADG_KERNEL_VOLSURF:
      return with_vol_shape<DIM, N, CURVED>(c, K, [&](auto s) {
        using S = decltype(s);
        using C = VolPairsCfg<DIM, N, CURVED, S::W, S::RR, S::HH>;
        *E = C::EB;
        *grid = vol_grid<C>(K);
        return (int)WADG_OK;
      });
    case WADG_KERNEL_SURF:
      *E = SurfMmaCfg<DIM, N>::EW;
      *grid = (K + *E - 1) / *E;
      return WADG_OK;
    case WADG_KERNEL_UPDATE:
      *E = UpdMmaCfg<DIM, N, CURVED>::EW;
      return update_grid<DIM, N, CURVED>(K, grid);
    case WADG_KERNEL_ADJ_PAIRS:
      return wadg_internal::adj_pairs_shape(DIM, N, CURVED, K, E, grid);
    case WADG_KERNEL_STAGE:
      return with_stage_warps<DIM, N, CURVED>(K, [&](auto w) {
        using C = VolPairsCfg<DIM, N, CURVED, decltype(w)::value>;
        *E = C::E;
        *grid = persistent_grid(K, C::E, C::smem_vol);
        return (int)WADG_OK;
      });
  }
  return fail(WADG_ERR_INVALID, "unknown kernel %d", kernel);
}

// Meshes of few groups take the wide shape: up to one group per SM in 3D, three
// in 2D.  Update kernel, us, default -> wide, by groups per SM: 3D N=2 0.1 5.5 ->
// 4.0, 2.6 6.5 -> 7.3; N=3 0.3 6.9 -> 5.4, 1.1 7.9 -> 8.9; curved N=4 0.6 13.8 -> 11.6,
// 1.7 20.0 -> 21.4; 2D N=3 1.7 4.6 -> 4.2, 2.7 5.0 -> 4.4, 6.9 7.6 -> 7.9.  Between events
// (some 4 us more), 2D: N=1, 2 no difference up to 9.7; N=3 1.7 9.7 -> 8.6, 3.9 10.2 -> 9.7,
// 5.2 11.8 -> 12.4; curved N=4 1.0 10.5 -> 9.8, 2.9 11.9 -> 11.9, 5.2 13.9 -> 17.8; 3D N=2 1.7
// 10.4 -> 9.8 (not taken), 2.6 10.4 -> 12.3
template <int DIM, int N, bool CURVED>
bool wide_update(int K) {
  return K <= (DIM == 3 ? 1 : 3) * num_sms() * UpdMmaCfg<DIM, N, CURVED>::EW;
}

template <int DIM, int N, bool CURVED, bool WIDE>
int launch_update_w(const wadg_ctx *c, int K, int grid, const double *Jq, const double *VqPq,
                    const double *VfPq, double fa, double fb, double fdt, double *rhsQ, double *resQ,
                    double *Q, double *Qf, const double *dtK, const int *glist, const int *ng) {
  using C = UpdMmaCfg<DIM, N, CURVED, WIDE>;
  // (update_grid raises the limit of the default shape's kernel, not of the wide one's)
  static_assert(C::smem <= (WIDE ? 48 : 227) * 1024, "update kernel does not fit in shared memory");
  return launch(c, "update kernel", overlaps<DIM, N>(c, K), update_mma_kernel<DIM, N, CURVED, WIDE>, grid,
                C::threads, C::smem, K, Jq, VqPq, VfPq, fa, fb, fdt, rhsQ, resQ, Q, Qf, c->phys, dtK, glist, ng);
}

template <int DIM, int N, bool CURVED>
int launch_update(const wadg_ctx *c, int K, const double *Jq, const double *VqPq,
                  const double *VfPq, double fa, double fb, double fdt, double *rhsQ,
                  double *resQ, double *Q, double *Qf, const double *dtK = nullptr,
                  const int *glist = nullptr, const int *ng = nullptr) {
  int grid = 0;
  if (int r = update_grid<DIM, N, CURVED>(K, &grid)) return r;
  if (wide_update<DIM, N, CURVED>(K))
    return launch_update_w<DIM, N, CURVED, true>(c, K, grid, Jq, VqPq, VfPq, fa, fb, fdt, rhsQ, resQ, Q,
                                                 Qf, dtK, glist, ng);
  return launch_update_w<DIM, N, CURVED, false>(c, K, grid, Jq, VqPq, VfPq, fa, fb, fdt, rhsQ, resQ, Q,
                                                Qf, dtK, glist, ng);
}

// every launch of one (dim, N, curved), defined in wadg_k<dim><N>.cu
#define WADG_LAUNCHES(X, D, N, C)                                                                  \
  X template int launch_volsurf<D, N, C>(                                                          \
      const wadg_ctx *, int, const double *, const double *, const double *, const uint32_t *,     \
      const double *, const double *, const double *, const double *, const double *,              \
      const double *, const double *, const double *, const double *, double *, const int *,       \
      const int *);                                                                                \
  X template int launch_vol_pairs<D, N, C>(                                                        \
      const wadg_ctx *, int, const double *, const double *, const double *, const double *,       \
      const double *, const double *, const double *, const double *, const double *,              \
      const double *, const double *, double *, double *);                                         \
  X template int launch_stage<D, N, C>(                                                            \
      const wadg_ctx *, int, const double *, const double *, const double *, const uint32_t *,     \
      const double *, const double *, const double *, const double *, const double *,              \
      const double *, const double *, const double *, const double *, const double *, double,      \
      double, double, const double *, const double *, double *, double *, double *, double *);     \
  X template int launch_update<D, N, C>(const wadg_ctx *, int, const double *, const double *,     \
                                        const double *, double, double, double, double *,          \
                                        double *, double *, double *, const double *, const int *, \
                                        const int *);                                              \
  X template int kernel_shape<D, N, C>(const wadg_ctx *, int, int, int *, int *);                  \
  X template int vol_warps_candidates<D, N, C>(int *);                                             \
  X template int vol_shapes<D, N, C>(int *, int *);
#define WADG_LAUNCHES_DEGREE(X, D, N)                                                              \
  WADG_LAUNCHES(X, D, N, true)                                                                     \
  WADG_LAUNCHES(X, D, N, false)                                                                    \
  X template int launch_surf<D, N>(const wadg_ctx *, int, const double *, const uint32_t *,        \
                                   const double *, const double *, const double *, double *);

}  // namespace wadg
