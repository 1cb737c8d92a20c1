"""The launch shapes a solve takes by its size (no kb_set_tuning), on both
sides of each rule, against the oracle; and the device-built equilibrium on
velocity grids that are and are not products."""
import numpy as np
import pytest

import kitgpu
from kitgpu.solver import Handle, initial_cells, kb_config, wall_states
from cases import cavity, oracle_for, quadrant, rho_u_t_error, sod

pytestmark = pytest.mark.gpu

# grids of fewer than two CTAs per multiprocessor, of just more, with odd nu
# (one velocity per thread), and long enough for more than 4 rows per CTA
SHAPES = [("tiny", cavity(nx=9, ny=13, nu=12, nv=10)), ("tiny-odd", cavity(nx=20, ny=11, nu=13, nv=9)),
          ("pairs", cavity(nx=32, ny=33, nu=28, nv=28)), ("odd", cavity(nx=33, ny=30, nu=29, nv=28)),
          ("rows", quadrant(nx=66, ny=150, nu=28, nv=28, flux="kfvs")),
          ("rows-ugks", quadrant(nx=65, ny=130, nu=32, nv=32))]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("name,cfg", SHAPES, ids=[c[0] for c in SHAPES])
def test_default_shapes_against_oracle(gpu_lib, name, cfg, prec, tol):
    KS, ctr, *faces, t = kitgpu.initialize(cfg, precision=prec)
    orc = oracle_for(KS)
    dt = kitgpu.timestep(KS, ctr, 0.0)
    kitgpu.step(KS, ctr, dt, 3)
    orc.step(dt, 3)
    got, ref = ctr.handle.download(), orc.get_state()
    assert max(rho_u_t_error(got["prim"], ref[1])) < tol
    for k, x in (("h", ref[2]), ("b", ref[3])):
        assert np.max(np.abs(got[k] - x)) < tol * np.max(np.abs(x)), k


@pytest.mark.parametrize("prec,tol", [("fp64", 0.0), ("fp32", 1.05 * 2 ** -24)])
def test_equilibrium_on_any_velocity_grid(gpu_lib, prec, tol):
    """A velocity grid in another order is no product of abscissae: the same
    equilibrium, velocity by velocity, in all cells.  On either side the
    exponent x carries 2.5 roundings, so a value 2.5 x 2^-53, and 8 more
    roundings follow; FP32 rounds it once more (values near 1e-36 have the low
    halves of their products among the denormals: 5 % of a rounding)."""
    KS = kitgpu.solver_set(quadrant(nx=7, ny=6, nu=13, nv=10))
    vs = KS.vs
    u, v, w = (vs.flat(x) for x in (vs.u, vs.v, vs.weights))
    perm = np.random.default_rng(1).permutation(len(u))
    W, P = initial_cells(KS)
    out = []
    for order in (np.arange(len(u)), perm):
        h = Handle(kb_config(KS, prec), u[order], v[order], w[order])
        h.init_equilibrium(W, P)
        s = h.download()
        back = np.argsort(order)
        out.append((s["h"][:, back], s["b"][:, back]))
    l = P[:, 3:4]
    x = l * ((u[None] - P[:, 1:2]) ** 2 + (v[None] - P[:, 2:3]) ** 2)
    H = P[:, :1] * (l / np.pi) * np.exp(-x)
    tol += 2 * (2.5 * x.max() + 8) * 2 ** -53
    for a in out:
        for got, ref in zip(a, (H, H * KS.gas.K / (2.0 * l))):
            assert np.max(np.abs(got - ref) / ref) < tol


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("name,cfg", [("cavity", cavity(nx=21, ny=18, nu=12, nv=10)),
                                      ("cavity-bgk-odd", cavity(nx=9, ny=16, nu=13, nv=9, flux="ugks", coll="bgk")),
                                      ("line", sod(nx=37, nu=33, flux="kcu", bc="maxwell"))],
                         ids=["cavity", "cavity-bgk-odd", "line"])
def test_stages_one_by_one_equal_whole_steps(gpu_lib, name, cfg, prec):
    """A whole step takes the walls in the moment passes' launch, the timed
    stages launch them apart: the same sums, bit for bit."""
    out = []
    for timed in (False, True):
        KS, ctr, *faces, t = kitgpu.initialize(cfg, precision=prec)
        dt = kitgpu.timestep(KS, ctr, 0.0)
        ctr.handle.set_timing(timed)
        kitgpu.step(KS, ctr, dt, 4)
        out.append(ctr.handle.download())
    for k in ("w", "prim", "h", "b"):
        assert np.array_equal(out[0][k], out[1][k]), k


FACTORED = [("kcu-shakhov-walls", cavity(nx=9, ny=12, nu=11, nv=8)),
            ("ugks-bgk-extra", quadrant(nx=10, ny=7, nu=9, nv=12)),
            ("ugks-shakhov-extra", quadrant(nx=13, ny=9, nu=8, nv=13, coll="shakhov")),
            ("kfvs-bgk-walls", cavity(nx=8, ny=9, nu=10, nv=7, flux="kfvs", coll="bgk")),
            ("kfvs-shakhov-fix", quadrant(nx=17, ny=18, nu=8, nv=9, flux="kfvs", coll="shakhov", bc="fix", ng=0))]


@pytest.mark.parametrize("name,cfg", FACTORED, ids=[c[0] for c in FACTORED])
def test_factored_maxwellians_equal_exponentials(gpu_lib, name, cfg):
    """FP64: a velocity grid in another order is no product, so its update takes
    the exponentials where the ordered one takes products of factors: the same
    states to the FP64 form's 1e-12 after 6 steps."""
    KS = kitgpu.solver_set(cfg)
    vs = KS.vs
    u, v, w = (vs.flat(x) for x in (vs.u, vs.v, vs.weights))
    perm = np.random.default_rng(2).permutation(len(u))
    W, P = initial_cells(KS)
    out = []
    for order in (np.arange(len(u)), perm):
        h = Handle(kb_config(KS, "fp64"), u[order], v[order], w[order])
        h.init_equilibrium(W, P)
        for side, prim in enumerate(wall_states(KS)):
            if KS.set.boundary[side] == "maxwell":
                h.set_wall(side, prim)
        h.step(h.timestep(KS.set.cfl, 0.0, 1e9), 6)
        s = h.download()
        back = np.argsort(order)
        out.append((s["prim"], s["h"][:, back], s["b"][:, back]))
    assert max(rho_u_t_error(out[0][0], out[1][0])) < 1e-12
    for x, y in zip(out[0][1:], out[1][1:]):
        assert np.max(np.abs(x - y)) < 1e-12 * np.max(y)
