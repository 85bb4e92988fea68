"""The work that users of this solver have it do, as timed cases.

A case names a workload and how a program calls it; ``prepare`` makes what
such a program holds before the call (mesh, app or buffers, initial state on
the GPU or in pinned host memory), ``run`` is one pass through the public entry
points, ``exact`` the same pass in plain 64-bit torch.

Calls (the key ``call``):

  solve     an ``App`` solve whose initial state is on the device: Q0 is copied
            into the app's state, projected, and advanced by graph-replayed time
            steps (one solve of a parameter study, or a solve chained to another
            program on the GPU)
  host      the same solve from and to host buffers (``App.solve_host_q``): a
            host program's call
  kernels   the three kernels with the OKL argument lists on the caller's own
            device buffers, five stages (the reference's C driver with its
            kernel launches replaced)
  gradient  ``Adjoint.forward`` and ``Adjoint.reverse``: Q(T) and dJ/dQ0 of a
            checkpointed run
  ensemble  a batch of independent 2D solves, each with its own step

Workloads (the key ``flow``): the isentropic vortex on triangles, the
Taylor-Green vortex (``mach`` is its Mach number, 0.1 in the standard set-up) and
the density wave on tetrahedra.  ``curved`` selects the weight-adjusted kernels
(on a warped mesh).  ``nx``, ``ny``: quads per direction of the square, split in
two; ``n``: hexes per direction of the cube, split in six.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from scratch_wadge_b200 import adjoint as ADJ
from scratch_wadge_b200 import capi
from scratch_wadge_b200 import ensemble as ENS
from scratch_wadge_b200 import geometry_gpu as GG
from scratch_wadge_b200 import ic as IC
from scratch_wadge_b200 import mesh as M

GAMMA = 1.4


def listed():
    tri = dict(dim=2, flow="vortex", curved=False, variant="volsurf")
    tet = dict(dim=3, flow="taylor_green", curved=False, variant="volsurf", mach=0.1)
    wave = dict(dim=3, flow="density_wave", curved=True, variant="three_kernels")
    return [
        # the smallest instance of a 2D parameter study: launches and latency count
        dict(tri, name="tri_K200_N2", call="solve", nx=20, ny=5, N=2, steps=10),
        # the standard 2D vortex run, a short stretch of it
        dict(tri, name="tri_K2048_N3", call="solve", nx=32, ny=32, N=3, steps=10),
        # the same flow on the finest of the measured 2D meshes
        dict(tri, name="tri_K32768_N3", call="solve", nx=128, ny=128, N=3, steps=10),
        # warped triangles of the highest degree, an element count no batch divides,
        # in the app's default stage (the three kernels)
        dict(tri, name="tri_curved_K2146_N4", call="solve", nx=37, ny=29, N=4, steps=10, curved=True,
             variant="three_kernels"),
        # a coarse 3D run in the app's default stage
        dict(tet, name="tet_K162_N2", call="solve", n=3, N=2, steps=10, variant="three_kernels"),
        # the Taylor-Green run the solver is quoted on
        dict(tet, name="tet_K24576_N3", call="solve", n=16, N=3, steps=5),
        # a solve called from a host program, odd element count, lower degree
        dict(tet, name="tet_host_K7986_N2", call="host", n=11, N=2, steps=20),
        # the density wave on warped tetrahedra, the highest degree
        dict(wave, name="tet_curved_K10368_N4", call="solve", n=12, N=4, steps=2),
        # warped tetrahedra, middle degree, an odd mesh
        dict(wave, name="tet_curved_K2058_N3", call="solve", n=7, N=3, steps=5, variant="volsurf"),
        # a C driver's kernel launches, a faster flow
        dict(tet, name="tet_kernels_K4374_N4", call="kernels", n=9, N=4, steps=1, mach=0.3,
             variant="three_kernels"),
        # the gradient of a Taylor-Green run on the mesh the adjoint is quoted on
        dict(tet, name="tet_gradient_K3072_N3", call="gradient", n=8, N=3, steps=20, every=5),
        # independent 2D solves of mixed size and degree, batched
        dict(name="ensemble_24", call="ensemble", dim=2, count=24, kmin=200, kmax=8192, mix=0, T=0.01),
    ]


def draw(rng):
    """One more case of the same ranges: the calls, flows, degrees, stage
    variants and sizes of the listed ones."""
    logint = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    call = rng.choice(["solve", "solve", "solve", "solve", "host", "kernels", "gradient", "ensemble"])
    if call == "ensemble":
        kmax = logint(1000, 8192)
        return dict(call=call, dim=2, count=rng.randint(5, 24), kmin=200, kmax=kmax,
                    mix=rng.randint(1, 10 ** 6), T=0.01)
    c = dict(call=call, dim=rng.choice([2, 3]), N=rng.randint(2, 4), curved=rng.random() < 0.4,
             variant="three_kernels" if call == "kernels" else rng.choice(["three_kernels", "volsurf"]))
    if c["dim"] == 2:
        K = logint(200, 32768)
        c["ny"] = max(3, int(round(math.sqrt(K / 2.0 * rng.uniform(0.4, 1.2)))))
        c["nx"] = min(128, max(3, int(round(K / (2.0 * c["ny"])))))
        c["ny"] = min(128, c["ny"])
        c["flow"] = "vortex"
    else:
        cells = logint(27, {2: 4096, 3: 4096, 4: 1728}[c["N"]])
        c["n"] = max(3, int(round(cells ** (1.0 / 3.0))))
        c["flow"] = "density_wave" if c["curved"] else rng.choice(["taylor_green", "density_wave"])
        if c["flow"] == "taylor_green":
            c["mach"] = round(rng.uniform(0.1, 0.5), 3)
    if call == "gradient":
        if c["dim"] == 3:
            c["n"] = min(c["n"], {2: 11, 3: 8, 4: 6}[c["N"]])
        else:
            c["nx"], c["ny"] = min(c["nx"], 64), min(c["ny"], 64)
        c["steps"] = rng.randint(4, 12)
        c["every"] = rng.randint(2, 5)
    elif call == "kernels":
        c["steps"] = 1
    else:
        big = c["dim"] == 3 and c["n"] > 8
        c["steps"] = rng.randint(2, 3) if big else rng.randint(5, 20)
    return c


# ------------------------------------------------------------------ inputs
def _warp2(x, y):
    w = 0.1 * np.sin(math.pi * x / 10.0) * np.cos(math.pi * y / 10.0)
    return x + w, y - 0.5 * w


@functools.lru_cache(maxsize=3)
def _geometry(dim, a, b, N, curved):
    """A program builds its mesh once; the initial states vary."""
    if dim == 2:
        mesh = M.periodic_square(a, b)
        if curved:
            mesh.warp = _warp2
    else:
        mesh = M.periodic_cube(a, warp=M.warp_cube(0.05) if curved else None)
    return GG.build_geometry_gpu(mesh, N)


def _geo(c):
    return _geometry(c["dim"], c["nx"] if c["dim"] == 2 else c["n"], c.get("ny", 0), c["N"], c["curved"])


def _initial(c, geo, seed):
    """Q0 [K][Nfields][Nq]: the flow's initial state with seeded parameters,
    L2-projected at the quadrature points."""
    rng = np.random.default_rng(seed)
    x = geo.xyzq.transpose(1, 0, 2)  # (3, K, Nq)
    if c["flow"] == "vortex":
        U = IC.vortex_2d(x[0], x[1], 0.0, GAMMA, beta=rng.uniform(3.0, 6.0), x0=rng.uniform(4.0, 16.0),
                         y0=rng.uniform(-2.0, 2.0))
    elif c["flow"] == "density_wave":
        U = IC.density_wave(x[0], x[1], x[2], rng.uniform(0.0, 2.0), GAMMA)
    else:
        s = rng.uniform(-math.pi, math.pi, 3)
        U = IC.taylor_green(x[0] + s[0], x[1] + s[1], x[2] + s[2], GAMMA)
        U[4] += (1.0 / c["mach"] ** 2 - 100.0) / (GAMMA * (GAMMA - 1.0))
    return np.ascontiguousarray((U @ geo.ops.VqPq.T).transpose(1, 0, 2))


def _dt(geo, Q0, N):
    return IC.time_step(geo, 0.5, N, wave_speed=IC.max_wave_speed(Q0))[0]


class _View:
    """Device memory of `owner`, which lives as long as a tensor over it."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8", data=(ptr, False),
                                             version=3)


def _state(app, owner=None):
    """The app's state arrays as tensors (no copy); owner: what frees the app."""
    p = app.state_ptrs()
    view = lambda k: _View(p[k], app.fshape if k == "Qf" else app.vshape, (app, owner))
    return {k: torch.as_tensor(view(k), device="cuda") for k in ("Q", "rhsQ", "Qf", "resQ")}


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _instances(c, seed):
    """Element counts and degrees from the case, vortices from the seed."""
    rng = np.random.default_rng(seed)
    got = ENS.draw_instances(c["count"], c["kmin"], c["kmax"], seed=c["mix"])
    for i in got:
        i.beta, i.x0, i.y0 = rng.uniform(3.0, 6.0), rng.uniform(0.0, 20.0), rng.uniform(-5.0, 5.0)
    return got


@functools.lru_cache(maxsize=32)
def _square(nx, ny, N):
    return M.build_geometry(M.periodic_square(nx, ny), N)


def _parts(instances):
    return [ENS.build_instance(i, GAMMA, builder=lambda mesh, N, i=i: _square(i.nx, i.ny, N))
            for i in instances]


def prepare(case, seed):
    c = case
    if c["call"] == "ensemble":
        inst = _instances(c, seed)
        ens = ENS.Ensemble(inst, parts=_parts(inst), T=c["T"], gamma=GAMMA)
        bins = []
        for b in ens.bins.values():
            init = {k: torch.from_numpy(b["state"][k]).cuda() for k in ("Q", "rhsQ", "Qf", "resQ")}
            bins.append((_state(b["app"], ens), init))
        return dict(call="ensemble", ens=ens, bins=bins)
    geo = _geo(c)
    Q0 = _initial(c, geo, seed)
    dt = _dt(geo, Q0, c["N"])
    s = dict(call=c["call"], dt=dt, steps=c["steps"])
    if c["call"] == "kernels":
        ops = geo.ops
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        col = lambda a: dev(np.asarray(a).T)  # column-major
        f = {k: dev(getattr(geo, k)) for k in ("vgeo", "vfgeo", "fgeo", "Jq")}
        f["mapPq"] = dev(geo.mapPq.view(np.int32))
        f.update({k: dev(getattr(ops, k)) for k in ("nrJ", "nsJ") + (("ntJ",) if c["dim"] == 3 else ())})
        f.update({k: col(getattr(ops, k)) for k in ("Drq", "Dsq", "VqLq", "VqPq", "VfPq") +
                  (("Dtq",) if c["dim"] == 3 else ())})
        Nf, f64 = ops.Nfields, dict(dtype=torch.float64, device="cuda")
        f.update({k: torch.zeros((geo.K, Nf, ops.Nq), **f64) for k in ("Q", "rhsQ", "resQ")})
        f.update({k: torch.zeros((geo.K, Nf, ops.NfqNf), **f64) for k in ("Qf", "rhsQf")})
        ctx = capi.Context(ops, GAMMA, stream=_stream().cuda_stream)
        s.update(ctx=ctx, f=f, p={k: t.data_ptr() for k, t in f.items()}, K=geo.K, curved=c["curved"],
                 Q0=dev(Q0))
        return s
    app = capi.App(geo, c["curved"], GAMMA, stream=_stream().cuda_stream)
    app.set_stage_variant(c["variant"])
    s.update(app=app)
    if c["call"] == "host":
        s.update(Q0=_pinned(Q0.shape), out=_pinned(Q0.shape))
        s["Q0"][...] = Q0
    else:
        # (the residual register is no result: the first coefficient of a step is 0)
        state = _state(app)
        s.update(Q0=torch.from_numpy(Q0).cuda(), state={k: state[k] for k in ("Q", "rhsQ", "Qf")})
    if c["call"] == "gradient":
        s.update(adj=ADJ.Adjoint(app, c["steps"], c["every"]),
                 w=torch.from_numpy(geo.ops.wq[None, :] * geo.Jq).cuda())
    return s


# ------------------------------------------------------------------ a pass
def run(s):
    call = s["call"]
    if call == "solve":
        app = s["app"]
        with torch.cuda.stream(_stream()):
            s["state"]["Q"].copy_(s["Q0"])
        app.project()
        app.rk_run(s["dt"], s["steps"], graph=True)
        return s["state"]
    if call == "host":
        return s["app"].solve_host_q(s["Q0"], s["dt"], s["steps"], out=s["out"])
    if call == "kernels":
        return _run_kernels(s)
    if call == "gradient":
        QT = s["adj"].forward(s["Q0"], s["dt"])
        bar = torch.zeros_like(QT)
        bar[:, 0, :] = 2.0 * s["w"] * QT[:, 0, :]  # J = int rho(T)^2
        return dict(QT=QT, Qbar0=s["adj"].reverse(bar))
    for state, init in s["bins"]:
        for k in init:
            state[k].copy_(init[k])
    torch.cuda.current_stream().synchronize()
    capi.check(capi.lib().wadg_ensemble_restart(s["ens"].h), "ensemble_restart")
    s["ens"].run()
    return [state["Q"] for state, _ in s["bins"]]


def _run_kernels(s):
    ctx, K, cv, p, f = s["ctx"], s["K"], s["curved"], s["p"], s["f"]
    g = p.get
    with torch.cuda.stream(_stream()):
        f["Q"].copy_(s["Q0"])
        f["rhsQ"].zero_()
    up = lambda curved, a, b, dt: ctx.update(curved, K, p["Jq"], p["VqPq"], p["VfPq"], a, b, dt,
                                             p["rhsQ"], p["resQ"], p["Q"], p["Qf"])
    up(False, 0.0, 0.0, 0.0)  # the stage-0 traces
    for _ in range(s["steps"]):
        for a, b in zip(IC.RK4A, IC.RK4B):
            ctx.vol(cv, K, p["vgeo"], p["vfgeo"], p["nrJ"], p["nsJ"], g("ntJ"), p["Drq"], p["Dsq"],
                    g("Dtq"), p["VqLq"], p["VfPq"], p["Qf"], p["rhsQ"], p["rhsQf"])
            ctx.surf(K, p["fgeo"], p["mapPq"], p["VqLq"], p["Qf"], p["rhsQf"], p["rhsQ"])
            up(cv, float(a), float(b), s["dt"])
    return {k: f[k] for k in ("Q", "rhsQ", "Qf")}


# ------------------------------------------------------------------ its work
def _sizes(dim, N):
    return {(2, 1): (3, 6), (2, 2): (6, 9), (2, 3): (12, 12), (2, 4): (16, 15),
            (3, 1): (4, 12), (3, 2): (11, 24), (3, 3): (23, 48), (3, 4): (44, 64)}[dim, N]


def _stage_flops(dim, N, curved):
    """One stage of one element: every two-point flux once (20 operations of
    the two log-means with their series, 6 per dimension and field to contract
    and to sum into both its rows), the lift, the inverse mass and the projection."""
    Nq, NF = _sizes(dim, N)
    Nf = dim + 2
    pairs = Nq * (Nq - 1) // 2 + Nq * NF + NF
    dense = 2 * Nf * (Nq * NF * 2 + Nq * Nq * (5 if curved else 2))
    return pairs * (30 + 6 * Nf + 4 * dim) + dense + 80 * (Nq + NF)


def work(case):
    c = case
    if c["call"] == "ensemble":
        flops = nbytes = 0.0
        for i in _instances(c, 0):
            Nq, NF = _sizes(2, i.N)
            # steps to T of an instance: dt = 0.5 hmin / C_N / wave speed (about 2)
            h = 20.0 / i.nx
            steps = max(1.0, c["T"] / (0.5 * 0.29 * h / ((i.N + 1) * (i.N + 2) / 2.0) / 2.0))
            flops += 5.0 * steps * i.K * _stage_flops(2, i.N, True)
            nbytes += 8.0 * i.K * (4 * Nq * 2 + (4 + 1) * Nq + (4 + 3) * NF)
        return dict(bytes=nbytes, flops=flops)
    dim, N = c["dim"], c["N"]
    K = 2 * c["nx"] * c["ny"] if dim == 2 else 6 * c["n"] ** 3
    Nq, NF = _sizes(dim, N)
    Nf, vgeo = dim + 2, dim * dim
    stages = 5.0 * c["steps"] * (3.0 if c["call"] == "gradient" else 1.0)
    geo = (vgeo * (Nq + NF) if c["curved"] else vgeo) + (dim + 1.5) * NF + Nq
    state = {"host": Nf * Nq, "gradient": 2 * Nf * Nq}.get(c["call"], Nf * (2 * Nq + NF))
    return dict(bytes=8.0 * K * (geo + Nf * Nq + state), flops=stages * K * _stage_flops(dim, N, c["curved"]))


# ------------------------------------------------------------------ 64 bits
class _Exact:
    """The stage map in plain torch, element chunks at a time."""

    def __init__(self, geo, curved):
        o = geo.ops
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()
        self.d, self.curved, self.K = o.dim, curved, geo.K
        d = self.d
        self.D = torch.stack([t(getattr(o, n)) for n in ("Drq", "Dsq", "Dtq")[:d]])
        self.Lq, self.Pq, self.Pf = t(o.VqLq), t(o.VqPq), t(o.VfPq)
        self.Nq, self.NF = o.Nq, o.NfqNf
        first = (np.arange(o.NfqNf) // o.Nfq) * o.Nfq
        self.nref = t(np.stack([np.asarray(getattr(o, n))[first] for n in ("nrJ", "nsJ", "ntJ")[:d]]))
        self.G = t(geo.vgeo).view(geo.K, d, d, o.Nq)
        self.Gf = t(geo.vfgeo).view(geo.K, d, d, o.NfqNf) if curved else None
        self.fg, self.J = t(geo.fgeo), t(geo.Jq)[:, None, :]
        m = np.asarray(geo.mapPq, dtype=np.int64).reshape(geo.K, -1)
        blk = o.NfqNf * o.Nfields
        self.mk, self.mj = (torch.from_numpy(a).cuda() for a in (m // blk, m % blk))
        self.chunk = max(1, 3_000_000 // (o.Nq * (o.Nq + o.NfqNf)))

    def project(self, Q, wadg):
        rho, m, E = Q[:, :1], Q[:, 1:-1], Q[:, -1:]
        e = E - 0.5 * (m * m).sum(1, keepdim=True) / rho
        s = torch.log((GAMMA - 1) * e) - GAMMA * torch.log(rho)
        V = torch.cat([(-E + e * (GAMMA + 1 - s)) / e, m / e, -rho / e], 1)
        if wadg:
            V = ((V * self.J) @ self.Pq.T / self.J) @ self.Pq.T

        def back(V):
            l, h = V[:, -1:], 0.5 * (V[:, 1:-1] ** 2).sum(1, keepdim=True) / V[:, -1:]
            lg = math.log(GAMMA - 1) - GAMMA * torch.log(-l) - (GAMMA - V[:, :1] + h)
            e = torch.exp(lg / (GAMMA - 1))
            return torch.cat([-e * l, e * V[:, 1:-1], e * (1 - h)], 1)

        return back(V @ self.Pq.T), back(V @ self.Pf.T)

    @staticmethod
    def mean(a, b):
        """Logarithmic mean: (a+b)/2 f / atanh f, f = (a-b)/(a+b)."""
        f = (a - b) / (a + b)
        u = f * f
        near = u < 1e-2
        ser = torch.full_like(u, 1.0 / 21)
        for k in range(9, -1, -1):
            ser = ser * u + 1.0 / (2 * k + 1)
        fs = torch.where(near, torch.full_like(f, 0.5), f)
        return 0.5 * (a + b) / torch.where(near, ser, 0.5 * (torch.log1p(fs) - torch.log1p(-fs)) / fs)

    def prim(self, U):
        rho, u = U[:, 0], U[:, 1:-1] / U[:, :1]
        p = (GAMMA - 1) * (U[:, -1] - 0.5 * rho * (u * u).sum(1))
        return rho, u, rho / (2 * p)

    def flux(self, A, B, n):
        """Entropy-conservative flux along n; a list of the fields."""
        (ra, ua, ba), (rb, ub, bb) = A, B
        rl, bl = self.mean(ra, rb), self.mean(ba, bb)
        pa = 0.5 * (ra + rb) / (ba + bb)
        av = [0.5 * (x + y) for x, y in zip(ua, ub)]
        un = sum(x * y for x, y in zip(av, n))
        kin = 0.5 * sum(x * y for x, y in zip(ua, ub))
        F0 = rl * un
        return [F0] + [F0 * x + pa * y for x, y in zip(av, n)] + \
            [(rl * (1 / (2 * (GAMMA - 1) * bl) + kin) + pa) * un]

    def rhs(self, uq, uf):
        d, out = self.d, []
        for z in range(0, self.K, self.chunk):
            k = slice(z, z + self.chunk)
            (rq, vq, bq), (rf, vf, bf) = self.prim(uq[k]), self.prim(uf[k])
            row = (rq[:, :, None], [vq[:, i, :, None] for i in range(d)], bq[:, :, None])
            colv = (rq[:, None, :], [vq[:, i, None, :] for i in range(d)], bq[:, None, :])
            colf = (rf[:, None, :], [vf[:, i, None, :] for i in range(d)], bf[:, None, :])
            G = self.G[k]
            nv, nf = [], []
            for x in range(d):
                if self.curved:
                    g = [0.5 * (G[:, a, x, :, None] + G[:, a, x, None, :]) for a in range(d)]
                    h = [0.5 * (G[:, a, x, :, None] + self.Gf[k][:, a, x, None, :]) for a in range(d)]
                else:
                    g = h = [G[:, a, x, :1, None] for a in range(d)]
                nv.append(sum(self.D[a] * g[a] for a in range(d)))
                nf.append(sum(self.nref[a] * h[a] for a in range(d)))
            F = self.flux(row, colf, nf)
            rows = [a.sum(2) + (0.5 * self.Lq * b).sum(2) for a, b in zip(self.flux(row, colv, nv), F)]
            face = torch.stack([(-0.5 * self.Pf.T * b).sum(1) for b in F], 1)
            UM, UP = uf[k], uf[self.mk[k], :, self.mj[k]].transpose(1, 2)
            rP, vP, bP = self.prim(UP)
            nJ, sJ = [self.fg[k, x] for x in range(d)], self.fg[k, d]
            Fs = self.flux((rf, list(vf.unbind(1)), bf), (rP, list(vP.unbind(1)), bP), nJ)
            lam = lambda v, b: torch.sqrt((v * v).sum(1)) + torch.sqrt(0.5 * GAMMA / b)
            L = 0.25 * torch.maximum(lam(vf, bf), lam(vP, bP)) * sJ
            sf = face + 0.5 * torch.stack(torch.broadcast_tensors(*Fs), 1) - L[:, None] * (UP - UM)
            out.append(torch.stack(rows, 1) + sf @ self.Lq.T)
        return torch.cat(out)

    def minv(self, r):
        r = -2.0 * (r @ self.Pq.T) / self.J
        return r @ self.Pq.T if self.curved else r

    def run(self, Q, dt, steps, each=None):
        res = torch.zeros_like(Q)
        uq, uf = self.project(Q, False)
        for _ in range(steps):
            for a, b in zip(IC.RK4A, IC.RK4B):
                if each is not None:
                    each.append(Q)
                res = a * res + dt * self.minv(self.rhs(uq, uf))
                Q = Q + b * res
                uq, uf = self.project(Q, self.curved)
        return dict(Q=Q, rhsQ=uq, Qf=uf)


def _exact_gradient(c, geo, Q0, dt):
    E, stages = _Exact(geo, c["curved"]), []
    # a checkpointed run projects every stage, the first too, with the stage's projection
    first = E.project
    E.project = lambda Q, wadg: first(Q, E.curved)
    with torch.no_grad():
        QT = E.run(Q0, dt, c["steps"], stages)["Q"]
    w = torch.from_numpy(geo.ops.wq[None, :] * geo.Jq).cuda()
    Qb, rb = torch.zeros_like(QT), torch.zeros_like(QT)
    Qb[:, 0, :] = 2.0 * w * QT[:, 0, :]
    for idx in range(len(stages) - 1, -1, -1):
        a, b = IC.RK4A[idx % 5], IC.RK4B[idx % 5]
        r = rb + b * Qb
        rb = a * r
        Q = stages[idx].detach().requires_grad_(True)
        R = E.minv(E.rhs(*E.project(Q, True)))
        Qb = Qb + torch.autograd.grad(R, Q, dt * r)[0]
    return dict(QT=QT, Qbar0=Qb)


def exact(case, seed):
    c = case
    if c["call"] == "ensemble":
        inst = _instances(c, seed)
        parts = _parts(inst)
        steps = ENS.instance_steps(parts, c["T"])
        got = {}
        with torch.no_grad():
            for i, (geo, st), (dt, n) in zip(inst, parts, steps):
                got.setdefault(i.N, []).append(_Exact(geo, True).run(torch.from_numpy(st["Q"]).cuda(), dt, n)["Q"])
        return [torch.cat(got[N]) for N in sorted(got)]
    geo = _geo(c)
    Q0 = _initial(c, geo, seed)
    dt = _dt(geo, Q0, c["N"])
    Q0 = torch.from_numpy(Q0).cuda()
    if c["call"] == "gradient":
        pairs = geo.K * geo.ops.Nq * (geo.ops.Nq + geo.ops.NfqNf)
        return _exact_gradient(c, geo, Q0, dt) if pairs < 12_000_000 else None
    with torch.no_grad():
        got = _Exact(geo, c["curved"]).run(Q0, dt, c["steps"])
    return got["Q"] if c["call"] == "host" else got
