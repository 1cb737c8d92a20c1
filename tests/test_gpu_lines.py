"""Single 1D solves that step in the fused segment kernels: what a call returns
beside the state."""
import numpy as np
import pytest

import kitgpu
from cases import oracle_for, shock, sod

pytestmark = pytest.mark.gpu

# one stepped cell, whole segments of each length and one cell more or less,
# ghosts (whose end faces are computed too) and none
LINES = [("three", sod(nx=3, nu=9)), ("three-ghosts", shock(nx=3, nu=12, ng=1)), ("four", sod(nx=4, nu=33)),
         ("six", shock(nx=6, nu=20, ng=2)), ("seven", sod(nx=7, nu=17, coll="bgk", ng=1)),
         ("ghosts", shock(nx=31, nu=33, ng=2)), ("plain", sod(nx=64, nu=49)), ("long", sod(nx=157, nu=40, ng=1))]


def _both(cfg, prec):
    KS, ctr, *faces, t = kitgpu.initialize(cfg, precision=prec)
    KS.set.maxTime = 1e9
    return KS, ctr, faces, oracle_for(KS), kitgpu.timestep(KS, ctr, 0.0)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5)])
@pytest.mark.parametrize("name,cfg", LINES, ids=[c[0] for c in LINES])
@pytest.mark.parametrize("how", ["solve", "step", "async", "cfl"])
def test_face_moments_of_the_last_step(gpu_lib, how, name, cfg, prec, tol):
    """fw after a call is that of its last step, on every face that has one."""
    KS, ctr, faces, orc, dt = _both(cfg, prec)
    n = 5 if how != "step" else 41  # graphs of 16 steps and single ones
    orc.step(dt, n - 1)
    orc.reconstruct()
    orc.evolve(dt)
    if how == "solve":
        KS.set.maxTime = (n - 0.5) * dt
        kitgpu.solve(KS, ctr, *faces)
        fw = faces[0].fluxes()[0]
    else:
        if how == "step":
            ctr.handle.step(dt, n)
        elif how == "async":
            ctr.handle.step_async(dt, n)
        else:
            ctr.handle.step(dt, n - 1)
            ctr.handle.step_cfl(2.0 * KS.set.cfl, 0.0, dt, 3)  # one step, to the end time
        fw = ctr.handle.faces(dt)[0]
    ref = orc.faces()[0]
    assert np.max(np.abs(ref)) > 0.0
    for k in range(3):
        # the sum of a face that has no flux of its own is rounding of its terms
        s = max(np.max(np.abs(ref[:, k])), 0.1 * np.max(np.abs(ref)))
        assert np.max(np.abs(fw[:, k] - ref[:, k])) < tol * s, k
