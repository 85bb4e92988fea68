"""The persistent kernels over several batches per CTA, against the oracle.

The volume, volume + surface, update and fused stage kernels (and the
adjoint's pair VJP kernel) launch at most as many CTAs as are resident at once; CTA b then takes
batches b, b + grid, b + 2 grid, ...  Small meshes never leave the first
batch, so each case here takes the kernel's own launch shape
(wadg_kernel_shape) and runs it on K = 2 * grid * E + r elements with
0 < r < E: CTA 0 runs three batches, the last one partial (its elements past
the end replicate element K-1 and are not stored).  That exercises the
prefetch of the next batch's traces, the per-group barriers across batches and
the partial-batch clamp.  Every compiled degree, affine and curved, 2D and 3D,
and every compiled CTA shape of the volume kernel, compared with the
reference's own kernels (oracle/_ref; the C restatement where it is absent)
at 1e-12.  The kernels run over the first K elements of larger arrays, so the
elements past K must come back untouched."""

import dataclasses
import math

import numpy as np
import pytest
import torch

from oracle import pyoracle as O
from oracle.torch_rhs import TorchRHS
from scratch_wadge_b200 import capi
from scratch_wadge_b200 import ic as IC
from scratch_wadge_b200 import mesh as M
from scratch_wadge_b200 import refops as R
from scratch_wadge_b200.adjoint import Adjoint
from scratch_wadge_b200.geometry_gpu import build_geometry_gpu
from tests.helpers import RTOL, perturbed, rel
from tests.test_gpu_parity import Dev

pytestmark = pytest.mark.gpu

CASES = [(d, N, c) for d in (2, 3) for N in (1, 2, 3, 4) for c in (False, True)]
SENTINEL = 12345.0


def oracle(ops, curved):
    """the reference's kernels where oracle/_ref was built, else the restatement"""
    try:
        return O.Reference(ops, curved)
    except FileNotFoundError:
        return O.Port(ops, curved)


def multibatch_K(E, grid):
    """2 * grid batches plus a partial one: CTA 0 runs three batches"""
    return 2 * grid * E + max(1, E // 3)


def mesh_with_at_least(dim, curved, K):
    if dim == 3:
        n = max(2, math.ceil((K / 6.0) ** (1.0 / 3.0)))
        return M.periodic_cube(n, warp=M.warp_cube(0.05) if curved else None)
    n = max(2, math.ceil(math.sqrt(K / 2.0)))
    return M.periodic_square(n, n)


def state(geo, curved, seed):
    """the stage-0 state of the case's flow, perturbed by 1% so that the
    log-mean's node pairs fall on both sides of its series switch"""
    dim = geo.ops.dim
    kind = "vortex" if dim == 2 else ("density_wave" if curved else "taylor_green")
    st = dict(zip(("Q", "rhsQ", "Qf", "resQ"), IC.stage0(geo, IC.initial_state(geo, kind))))
    st = perturbed(st, seed)
    st["resQ"] = 1e-3 * st["Q"]
    st["rhsQf"] = np.full_like(st["Qf"], SENTINEL)
    return st


def without_last_element(geo):
    """the mesh but its last element, whose neighbours' faces see themselves"""
    K, per = geo.K - 1, geo.ops.NfqNf * geo.ops.Nfields
    own = (np.arange(K)[:, None] * per + np.arange(geo.ops.NfqNf)[None, :]).reshape(geo.mapPq[:K].shape)
    mapPq = np.where(geo.mapPq[:K] // per == K, own, geo.mapPq[:K]).astype(np.uint32)
    cut = {k: np.ascontiguousarray(getattr(geo, k)[:K]) for k in ("vgeo", "vfgeo", "fgeo", "Jq", "xyzq", "xyzf")}
    return dataclasses.replace(geo, K=K, mapPq=mapPq, **cut)


def shapes(ctx, curved, K):
    """per volume kernel shape: ((warps, rows), E, grid at K)"""
    out = []
    for w, r in ctx.vol_shapes(curved):
        ctx.set_vol_shape(curved, w, r)
        out.append(((w, r),) + ctx.shape("vol", curved, K))
    ctx.set_vol_warps(curved, 0)
    return out


def _first(st, K):
    return {k: np.ascontiguousarray(v[:K]).copy() for k, v in st.items()}


@pytest.mark.parametrize("dim,N,curved", CASES)
def test_kernels_over_several_batches_per_cta(cuda, dim, N, curved):
    ops = R.load(dim, N)
    ctx = capi.Context(ops)
    big = 1 << 22  # the grid no longer grows with K beyond this
    sh = shapes(ctx, curved, big)
    Ku_E, Ku_g = ctx.shape("update", curved, big)
    Ks_E, Ks_g = ctx.shape("stage", curved, big)
    Kvs_E, Kvs_g = ctx.shape("volsurf", curved, big)
    Kvol = {w: multibatch_K(E, g) for w, E, g in sh}
    Kupd, Kst, Kvs = multibatch_K(Ku_E, Ku_g), multibatch_K(Ks_E, Ks_g), multibatch_K(Kvs_E, Kvs_g)
    mesh = mesh_with_at_least(dim, curved, max(max(Kvol.values()), Kupd, Kst, Kvs))
    geo = build_geometry_gpu(mesh, N)
    d = Dev(cuda, geo, curved)
    ref = oracle(ops, curved)
    st = state(geo, curved, 5)
    # a stable step for the mesh (the finer the mesh, the smaller), so that
    # the update of these rough states stays physical
    dt = IC.time_step(geo, 0.1, N, nsteps=1, wave_speed=IC.max_wave_speed(st["Q"]))[0]

    # volume kernel, every compiled shape
    for w, E, g in sh:
        K = Kvol[w]
        assert (K + E - 1) // E > 2 * g and K % E, (w, E, g, K)
        d.ctx.set_vol_shape(curved, *w)
        s = d.put(st)
        d.ctx.vol(curved, K, *[d.g[n].data_ptr() for n in ("vgeo", "vfgeo", "nrJ", "nsJ", "ntJ", "Drq",
                                                           "Dsq", "Dtq", "VqLq", "VfPq")],
                  s["Qf"].data_ptr(), s["rhsQ"].data_ptr(), s["rhsQf"].data_ptr())
        d.sync()
        h = d.get(s)
        a = _first(st, K)
        ref.vol(geo, a["Qf"], a["rhsQ"], a["rhsQf"])
        assert rel(h["rhsQ"][:K], a["rhsQ"]) < RTOL, (w, rel(h["rhsQ"][:K], a["rhsQ"]))
        assert rel(h["rhsQf"][:K], a["rhsQf"]) < RTOL, (w, rel(h["rhsQf"][:K], a["rhsQf"]))
        assert np.array_equal(h["rhsQ"][K:], st["rhsQ"][K:]), w
        assert (h["rhsQf"][K:] == SENTINEL).all(), w
    d.ctx.set_vol_warps(curved, 0)

    # surface (one CTA per group, not persistent) and update over Kupd elements
    K = Kupd
    s = d.put(st)
    rhsQf = st["Qf"] * 0.01  # stands in for the volume kernel's face rows
    s["rhsQf"] = torch.from_numpy(rhsQf).cuda()
    d.ctx.surf(K, d.g["fgeo"].data_ptr(), d.g["mapPq"].data_ptr(), d.g["VqLq"].data_ptr(),
               s["Qf"].data_ptr(), s["rhsQf"].data_ptr(), s["rhsQ"].data_ptr())
    d.ctx.update(curved, K, d.g["Jq"].data_ptr(), d.g["VqPq"].data_ptr(), d.g["VfPq"].data_ptr(),
                 IC.RK4A[2], IC.RK4B[2], dt, s["rhsQ"].data_ptr(), s["resQ"].data_ptr(),
                 s["Q"].data_ptr(), s["Qf"].data_ptr())
    d.sync()
    h = d.get(s)
    a = _first(dict(st, rhsQf=rhsQf), K)
    # the surface kernel gathers neighbour traces past K: give the oracle the
    # whole trace array, updating only the first K elements
    Qf_all = np.ascontiguousarray(st["Qf"]).copy()
    ref.surf(geo, Qf_all, a["rhsQf"], a["rhsQ"])
    ref.update(geo, IC.RK4A[2], IC.RK4B[2], dt, a["rhsQ"], a["resQ"], a["Q"], a["Qf"])
    for k in ("Q", "rhsQ", "Qf", "resQ"):
        assert np.isfinite(a[k]).all(), k
        assert rel(h[k][:K], a[k]) < RTOL, (k, rel(h[k][:K], a[k]))
        assert np.array_equal(h[k][K:], st[k][K:]), k

    # volume + surface kernel over Kvs elements (gathers traces past K)
    K = Kvs
    s = d.put(st)
    d.ctx.volsurf(curved, K, *[d.g[n].data_ptr() for n in ("vgeo", "vfgeo", "fgeo", "mapPq", "nrJ", "nsJ",
                                                           "ntJ", "Drq", "Dsq", "Dtq", "VqLq", "VfPq")],
                  s["Qf"].data_ptr(), s["rhsQ"].data_ptr())
    d.sync()
    h = d.get(s)
    a = _first(st, K)
    a["rhsQf"][:] = 0.0
    ref.vol(geo, a["Qf"], a["rhsQ"], a["rhsQf"])
    ref.surf(geo, np.ascontiguousarray(st["Qf"]).copy(), a["rhsQf"], a["rhsQ"])
    assert np.isfinite(a["rhsQ"]).all()
    assert rel(h["rhsQ"][:K], a["rhsQ"]) < RTOL, rel(h["rhsQ"][:K], a["rhsQ"])
    assert np.array_equal(h["rhsQ"][K:], st["rhsQ"][K:])
    assert np.array_equal(h["Qf"], st["Qf"])

    # fused stage kernel over Kst elements (reads the state, writes new buffers)
    K = Kst
    s = d.put(st)
    out = {"rhsQ": torch.full_like(s["rhsQ"], SENTINEL), "Qf": torch.full_like(s["Qf"], SENTINEL)}
    g = d.g
    fn = capi.lib().wadg_euler_stage_3d if dim == 3 else capi.lib().wadg_euler_stage_2d
    args = [g[n].data_ptr() for n in ("vgeo", "vfgeo", "fgeo", "mapPq", "nrJ", "nsJ")]
    args += [g["ntJ"].data_ptr()] if dim == 3 else []
    args += [g["Drq"].data_ptr(), g["Dsq"].data_ptr()] + ([g["Dtq"].data_ptr()] if dim == 3 else [])
    args += [g[n].data_ptr() for n in ("VqLq", "VfPq", "VqPq", "Jq")]
    capi.check(fn(d.ctx.h, K, int(curved), *args, IC.RK4A[3], IC.RK4B[3], dt, s["rhsQ"].data_ptr(),
                  s["Qf"].data_ptr(), s["Q"].data_ptr(), s["resQ"].data_ptr(), out["rhsQ"].data_ptr(),
                  out["Qf"].data_ptr()), "stage")
    d.sync()
    a = _first(st, K)
    a["rhsQf"][:] = 0.0
    Qf_all = np.ascontiguousarray(st["Qf"]).copy()
    ref.vol(geo, a["Qf"], a["rhsQ"], a["rhsQf"])
    ref.surf(geo, Qf_all, a["rhsQf"], a["rhsQ"])
    ref.update(geo, IC.RK4A[3], IC.RK4B[3], dt, a["rhsQ"], a["resQ"], a["Q"], a["Qf"])
    got = dict(Q=s["Q"].cpu().numpy(), resQ=s["resQ"].cpu().numpy(), rhsQ=out["rhsQ"].cpu().numpy(),
               Qf=out["Qf"].cpu().numpy())
    for k in ("Q", "rhsQ", "Qf", "resQ"):
        assert np.isfinite(a[k]).all(), k
        assert rel(got[k][:K], a[k]) < RTOL, (k, rel(got[k][:K], a[k]))
    assert np.array_equal(got["Q"][K:], st["Q"][K:])
    assert (got["rhsQ"][K:] == SENTINEL).all() and (got["Qf"][K:] == SENTINEL).all()


@pytest.mark.parametrize("dim,N,curved", [(3, 3, False), (3, 4, True), (2, 3, True)])
def test_adjoint_pair_kernel_over_several_batches(cuda, dim, N, curved):
    """the RHS VJP (pair kernel over several batches per CTA, a partial last
    batch) against reverse-mode autodiff of the restated stage map, run on the
    GPU through torch at this size"""
    ops = R.load(dim, N)
    ctx = capi.Context(ops)
    E, g = ctx.shape("adj_pairs", curved, 1 << 22)
    # the smallest structured mesh with more than 2 grid batches; where whole batches
    # tile it (E = 6 tiles every mesh of hexes cut in six), without its last element
    geo = build_geometry_gpu(mesh_with_at_least(dim, curved, 2 * g * E + 2), N)
    geo = geo if geo.K % E else without_last_element(geo)
    assert (geo.K + E - 1) // E > 2 * g and geo.K % E
    kind = "vortex" if dim == 2 else ("density_wave" if curved else "taylor_green")
    Q = perturbed({"Q": IC.stage0(geo, IC.initial_state(geo, kind))[0]}, 3, 1e-2)["Q"]
    w = np.random.default_rng(2).standard_normal(Q.shape)
    app = capi.App(geo, curved)
    adj = Adjoint(app, 1, 1)
    dev = torch.device("cuda")
    gq = adj.rhs_vjp(torch.from_numpy(Q).to(dev), torch.from_numpy(w).to(dev)).cpu().numpy()
    T = TorchRHS(geo, curved, device=dev)
    _, vjp = torch.func.vjp(T.R, torch.from_numpy(Q).to(dev))
    want = vjp(torch.from_numpy(w).to(dev))[0].cpu().numpy()
    assert rel(gq, want) < 1e-10, rel(gq, want)


@pytest.mark.parametrize("dim,N,curved", CASES)
def test_small_mesh_shape_edges(cuda, dim, N, curved):
    """Small meshes take another shape of the volume kernels (a warp per face of
    an element group): the smallest element counts, a partial last slice, the
    last count that takes it and the first that does not, against the
    reference's kernels."""
    ctx = capi.Context(R.load(dim, N))
    E1 = ctx.shape("volsurf", curved, 1)[0]
    lo, hi = 1, 1 << 20  # lo takes the small shape, hi does not
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if ctx.shape("volsurf", curved, mid)[0] == E1 else (lo, mid)
    assert 300 < lo < 1 << 16 and ctx.shape("vol", curved, lo)[0] == E1 != ctx.shape("vol", curved, hi)[0]
    geo = build_geometry_gpu(mesh_with_at_least(dim, curved, hi), N)
    d = Dev(cuda, geo, curved)
    ref = oracle(geo.ops, curved)
    st = state(geo, curved, 6)
    p = lambda s, *names: [s[n].data_ptr() for n in names]
    geom = ("vgeo", "vfgeo", "nrJ", "nsJ", "ntJ", "Drq", "Dsq", "Dtq", "VqLq", "VfPq")
    full = {k: v.copy() for k, v in st.items()}
    ref.vol(geo, full["Qf"], full["rhsQ"], full["rhsQf"])
    rows, faces = full["rhsQ"].copy(), full["rhsQf"].copy()
    ref.surf(geo, full["Qf"], full["rhsQf"], full["rhsQ"])
    for K in (1, 3, lo - 1, lo, hi):
        s = d.put(st)
        d.ctx.vol(curved, K, *p(d.g, *geom), *p(s, "Qf", "rhsQ", "rhsQf"))
        d.sync()
        h = d.get(s)
        assert rel(h["rhsQ"][:K], rows[:K]) < RTOL, (K, rel(h["rhsQ"][:K], rows[:K]))
        assert rel(h["rhsQf"][:K], faces[:K]) < RTOL, (K, rel(h["rhsQf"][:K], faces[:K]))
        assert np.array_equal(h["rhsQ"][K:], st["rhsQ"][K:]) and (h["rhsQf"][K:] == SENTINEL).all(), K
        s = d.put(st)
        d.ctx.volsurf(curved, K, *p(d.g, "vgeo", "vfgeo", "fgeo", "mapPq", *geom[2:]), *p(s, "Qf", "rhsQ"))
        d.sync()
        h = d.get(s)
        assert rel(h["rhsQ"][:K], full["rhsQ"][:K]) < RTOL, (K, rel(h["rhsQ"][:K], full["rhsQ"][:K]))
        assert np.array_equal(h["rhsQ"][K:], st["rhsQ"][K:]), K


def test_warps_by_rounds_curved_n2(cuda):
    """At curved 3D N=2 the volume and fused stage kernels take eight warps where
    twelve save no round: a partial batch, the last count of two rounds of eight
    and the first past it (twelve), against the reference's stage."""
    two = 2 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    geo = build_geometry_gpu(mesh_with_at_least(3, True, two + 1), 2)
    d = Dev(cuda, geo, True)
    st = state(geo, True, 5)
    dt = IC.time_step(geo, 0.1, 2, nsteps=1, wave_speed=IC.max_wave_speed(st["Q"]))[0]
    ref = oracle(geo.ops, True)
    want = _first(st, geo.K)
    want["rhsQf"][:] = 0.0
    ref.vol(geo, want["Qf"], want["rhsQ"], want["rhsQf"])
    ref.surf(geo, want["Qf"].copy(), want["rhsQf"], want["rhsQ"])
    rhs = want["rhsQ"].copy()
    ref.update(geo, IC.RK4A[3], IC.RK4B[3], dt, want["rhsQ"], want["resQ"], want["Q"], want["Qf"])
    names = ("vgeo", "vfgeo", "fgeo", "mapPq", "nrJ", "nsJ", "ntJ", "Drq", "Dsq", "Dtq", "VqLq", "VfPq",
             "VqPq", "Jq")
    for K, E in ((33, 32), (two, 32), (two + 1, 48)):
        assert d.ctx.shape("stage", True, K)[0] == E, K
        s = d.put(st)
        out = {k: torch.full_like(s[k], SENTINEL) for k in ("rhsQ", "Qf")}
        d.ctx.stage(True, K, *[d.g[n].data_ptr() for n in names], IC.RK4A[3], IC.RK4B[3], dt,
                    *[s[k].data_ptr() for k in ("rhsQ", "Qf", "Q", "resQ")], out["rhsQ"].data_ptr(),
                    out["Qf"].data_ptr())
        d.sync()
        h = d.get(dict(s, **out))
        for k in ("Q", "rhsQ", "Qf", "resQ"):
            assert rel(h[k][:K], want[k][:K]) < RTOL, (K, k, rel(h[k][:K], want[k][:K]))
        assert np.array_equal(h["Q"][K:], st["Q"][K:]) and (h["rhsQ"][K:] == SENTINEL).all(), K
        assert K == 33 or d.ctx.shape("volsurf", True, K)[0] == E, K
        s = d.put(st)
        d.ctx.volsurf(True, K, *[d.g[n].data_ptr() for n in names[:12]], s["Qf"].data_ptr(), s["rhsQ"].data_ptr())
        d.sync()
        h = d.get(s)
        assert rel(h["rhsQ"][:K], rhs[:K]) < RTOL and np.array_equal(h["rhsQ"][K:], st["rhsQ"][K:]), K


@pytest.mark.parametrize("dim,N,curved", CASES)
def test_small_mesh_cta_sizes(cuda, dim, N, curved):
    """A small mesh's CTA has 12 warps, or those of two slices where an SM has
    two: the element counts on either side of one and of two slices per SM give
    the same elements the same bits, and those of the reference's kernels."""
    ctx = capi.Context(R.load(dim, N))
    G = ctx.shape("volsurf", curved, 1)[0] // (12 // (dim + 1))
    one = G * torch.cuda.get_device_properties(0).multi_processor_count
    geo = build_geometry_gpu(mesh_with_at_least(dim, curved, 2 * one + 1), N)
    d = Dev(cuda, geo, curved)
    ref = oracle(geo.ops, curved)
    st = state(geo, curved, 9)
    want = {k: v.copy() for k, v in st.items()}
    ref.vol(geo, want["Qf"], want["rhsQ"], want["rhsQf"])
    faces = want["rhsQf"].copy()
    ref.surf(geo, want["Qf"], want["rhsQf"], want["rhsQ"])
    p = lambda s, *names: [s[n].data_ptr() for n in names]
    geom = ("vgeo", "vfgeo", "nrJ", "nsJ", "ntJ", "Drq", "Dsq", "Dtq", "VqLq", "VfPq")
    got = {}
    for K in (one - 1, one, one + 1, 2 * one - G, 2 * one, 2 * one + 1):
        s = d.put(st)
        d.ctx.vol(curved, K, *p(d.g, *geom), *p(s, "Qf", "rhsQ", "rhsQf"))
        d.sync()
        f = d.get(s)["rhsQf"]
        s = d.put(st)
        d.ctx.volsurf(curved, K, *p(d.g, "vgeo", "vfgeo", "fgeo", "mapPq", *geom[2:]), *p(s, "Qf", "rhsQ"))
        d.sync()
        r = d.get(s)["rhsQ"]
        assert rel(f[:K], faces[:K]) < RTOL and rel(r[:K], want["rhsQ"][:K]) < RTOL, K
        assert (f[K:] == SENTINEL).all() and np.array_equal(r[K:], st["rhsQ"][K:]), K
        got[K] = (f, r)
    whole = one - one % G - G  # slices that every count has whole
    for f, r in got.values():
        assert np.array_equal(f[:whole], got[one][0][:whole]) and np.array_equal(r[:whole], got[one][1][:whole])


@pytest.mark.parametrize("dim,N,curved", CASES)
def test_update_shape_edges(cuda, dim, N, curved):
    """The update kernel's two shapes (a warp per m-tile of the output projection
    on meshes of few groups): a single element, a partial group, and the last
    element count of the wide shape and the first past it, against the
    reference's kernel."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    last = (1 if dim == 3 else 3) * sms * 8
    geo = build_geometry_gpu(mesh_with_at_least(dim, curved, last + 1), N)
    d = Dev(cuda, geo, curved)
    st = state(geo, curved, 8)
    st["rhsQ"] = 1e-3 * st["rhsQ"]
    dt = IC.time_step(geo, 0.1, N, nsteps=1, wave_speed=IC.max_wave_speed(st["Q"]))[0]
    for K in (1, 9, last, last + 1):
        s = d.put(st)
        d.ctx.update(curved, K, *[d.g[n].data_ptr() for n in ("Jq", "VqPq", "VfPq")], IC.RK4A[1],
                     IC.RK4B[1], dt, *[s[n].data_ptr() for n in ("rhsQ", "resQ", "Q", "Qf")])
        d.sync()
        h = d.get(s)
        a = _first(st, K)
        oracle(geo.ops, curved).update(geo, IC.RK4A[1], IC.RK4B[1], dt, a["rhsQ"], a["resQ"], a["Q"], a["Qf"])
        for k in ("Q", "rhsQ", "Qf", "resQ"):
            assert np.isfinite(a[k]).all() and rel(h[k][:K], a[k]) < RTOL, (K, k, rel(h[k][:K], a[k]))
            assert np.array_equal(h[k][K:], st[k][K:]), (K, k)
