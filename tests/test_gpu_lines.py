"""Single 1D solves that step in the fused segment kernels: what a call returns
beside the state (face moments, residual, time), and where it stops."""
import numpy as np
import pytest

import kitgpu
from kitgpu._native import KitGPUError
from cases import oracle_for, rho_u_t_error, shock, sod

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


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_adaptive_steps_stop_at_a_state_that_is_not_physical(gpu_lib, prec):
    """A step far beyond the CFL limit leaves a negative density: the call fails,
    and the handle holds the state that step left, as after single steps."""
    out = []
    for n in (1, 20):
        KS, ctr, faces, orc, dt = _both(sod(nx=60, nu=33), prec)
        with pytest.raises(KitGPUError) as e:
            ctr.handle.step_cfl(40.0, 0.0, 1e9, n)
        assert e.value.code == -4
        out.append(ctr.handle.download())
    assert np.any(out[0]["prim"] <= 0.0)
    for k in ("w", "prim", "h", "b"):
        assert np.array_equal(out[0][k], out[1][k], equal_nan=True), k


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("stop", [0.3, 7.5, 66.2])
def test_end_time_inside_a_chunk(gpu_lib, stop, prec):
    """An end time before the last step of a call: the shorter last step, then the
    state is carried over; the time, state and residual of single steps."""
    KS, a, fa, orc, dt = _both(sod(nx=70, nu=36), prec)
    KS, b, fb, orc, dt = _both(sod(nx=70, nu=36), prec)
    end = stop * dt
    ta, ra = a.handle.step_cfl(KS.set.cfl, 0.0, end, 100)
    t, rb = 0.0, None
    while t < end * (1 - 1e-14):
        d = b.handle.timestep(KS.set.cfl, t, end)
        rb = b.handle.step(d, 1)
        t += d
    tol = 1e-12 if prec == "fp64" else 1e-5
    assert abs(ta - end) <= 1e-13 * end and abs(t - end) <= 1e-13 * end
    x, y = a.handle.download(), b.handle.download()
    assert max(rho_u_t_error(x["prim"], y["prim"])) < tol
    assert np.max(np.abs(x["h"] - y["h"])) < tol * np.max(y["h"])
    assert np.allclose(ra, rb, rtol=1e-9 if prec == "fp64" else 1e-4)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("name,cfg", LINES, ids=[c[0] for c in LINES])
def test_residual_is_the_change_of_w(gpu_lib, name, cfg, prec):
    """sqrt(sum dw^2 nx) / (sum |w| + 1e-7) of the FP64 w, dw and its sums in FP64
    in either precision of the distributions: nx roundings of terms of one
    sign, and a few of the root and quotient (1e-13)."""
    KS, ctr, faces, orc, dt = _both(cfg, prec)
    ctr.handle.step(dt, 4)
    before = ctr.handle.download()["w"]
    r = ctr.handle.step(dt, 1)
    after = ctr.handle.download()["w"]
    nx, ng = KS.ps.nx, ctr.handle.cfg.ngx
    i = slice(ng + 1, ng + nx - 1)  # the stepped cells
    dw = after[i] - before[i]
    want = np.sqrt(np.sum(dw * dw, 0) * nx) / (np.sum(np.abs(after[i]), 0) + 1e-7)
    assert np.all(np.abs(r - want) <= 1e-13 * want), (r, want)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_timed_steps_are_the_steps_of_a_solve(gpu_lib, prec):
    """Stage timing (kb_set_timing) of a line times the kernels that its solve
    runs: the same state and residual, bit for bit."""
    out = []
    for timed in (False, True):
        KS, ctr, faces, orc, dt = _both(sod(nx=37, nu=33), prec)
        ctr.handle.set_timing(timed)
        r = ctr.handle.step(dt, 5)
        if timed:
            st = ctr.handle.timing()
            assert all(n == 5 for _, n in st.values())
            assert sum(ms for ms, _ in st.values()) > 0.0
        s = ctr.handle.download()
        out.append((r, s["w"], s["prim"], s["h"], s["b"], ctr.handle.faces(dt)[0]))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("nx,nu", [(2048, 100), (5000, 33), (20011, 20)])
def test_long_lines_against_oracle(gpu_lib, nx, nu):
    """FP32 lines of more segments than the GPU holds at once."""
    KS, ctr, faces, orc, dt = _both(sod(nx=nx, nu=nu), "fp32")
    kitgpu.step(KS, ctr, dt, 8)
    orc.step(dt, 8)
    got, ref = ctr.handle.download(), orc.get_state()
    assert max(rho_u_t_error(got["prim"], ref[1])) < 1e-5
    for key, x in (("h", ref[2]), ("b", ref[3])):
        assert np.max(np.abs(got[key] - x)) < 1e-5 * np.max(np.abs(x)), key


def test_fp32_line_at_mach_8(gpu_lib):
    """500 steps of a single Mach 8 shock in the FP32 split form: rho, U and T
    within 1e-5 of FP64, as the ensembles' members."""
    st = []
    for prec in ("fp64", "fp32"):
        KS, ctr, *faces, t = kitgpu.initialize(shock(nx=100, nu=128, Ma=8.0, ng=0), precision=prec)
        if prec == "fp64":
            dt = kitgpu.timestep(KS, ctr, 0.0)
        kitgpu.step(KS, ctr, dt, 500)
        st.append(ctr.handle.download()["prim"])
    assert max(rho_u_t_error(st[1], st[0])) < 1e-5
