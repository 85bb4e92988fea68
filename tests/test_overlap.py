"""Kernels of the smallest meshes may start before their predecessor has ended
(programmatic dependent launch, in a captured time step): what a predecessor
writes is not constant while such a kernel runs, so it is neither declared nor
read as if it were, and a graph's steps equal the same launches one after
another bit for bit."""

import glob
import os
import re

import numpy as np
import pytest

from scratch_wadge_b200 import capi, ic as IC, mesh as M

CSRC = os.path.join(os.path.dirname(capi.__file__), "csrc")
WRITTEN = {"Q", "resQ", "rhsQ", "Qf", "rhsQf"}  # by the kernels of a stage


def overlapped_kernels():
    """{kernel: (parameter list, body)} of the kernels that wait for their predecessor"""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for part in src.split("__global__")[1:]:
            m = re.search(r"(\w+)\((int K,[^{]*)\)\s*\{", part)
            if m and "pdl_wait()" in part:
                out[m.group(1)] = (m.group(2), part[m.end():])
    return out


def test_what_a_predecessor_writes_is_not_declared_constant():
    kernels = overlapped_kernels()
    assert set(kernels) == {"vol_pairs_kernel", "surf_mma_kernel", "update_mma_kernel"}
    for name, (params, body) in kernels.items():
        decl = {re.search(r"(\w+)\s*(=.*)?$", p.strip()).group(1): p for p in params.split(",")}
        assert WRITTEN & set(decl), name
        for p in WRITTEN & set(decl):
            assert "__restrict__" not in decl[p], (name, p)
            assert not re.search(r"__ldg\(\s*%s\b" % p, body), (name, p)
    # the update kernel's staging of the right-hand side
    update = open(os.path.join(CSRC, "wadg_update_mma.cuh")).read()
    assert "__ldg(src" not in update


@pytest.mark.gpu
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("variant", ["three_kernels", "volsurf"])
def test_captured_steps_equal_launches_one_by_one(cuda, variant, dim, N, curved):
    mesh = M.periodic_square(20, 5) if dim == 2 else \
        M.periodic_cube(3, warp=M.warp_cube(0.05) if curved else None)
    geo = M.build_geometry(mesh, N)  # at most one element group per SM
    kind = "vortex" if dim == 2 else "density_wave" if curved else "taylor_green"
    Q0 = IC.stage0(geo, IC.initial_state(geo, kind, 1.4), 1.4)[0]
    dt = IC.time_step(geo, 0.5, N, wave_speed=IC.max_wave_speed(Q0))[0]
    got = []
    for graph in (True, False):
        app = capi.App(geo, curved)
        app.set_stage_variant(variant)
        app.set_state(Q=Q0)
        app.project()
        app.rk_run(dt, 20, graph=graph)
        got.append(app.get_state())
        app.close()
    for k in got[0]:
        assert np.isfinite(got[0][k]).all() and np.array_equal(got[0][k], got[1][k]), k
