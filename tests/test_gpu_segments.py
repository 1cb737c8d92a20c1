"""The fused segment kernels at the edges of their splits: segments of 3, 7, 15
and 31 cells, the chunks of cells a thread takes, velocity pairs, and the single
1D solves that take them (up to 256 velocities) against those that do not."""
import numpy as np
import pytest

import kitgpu
from kitgpu import batch as KB
from cases import oracle_for, rho_u_t_error, shock, sod

pytestmark = pytest.mark.gpu

# one stepped cell, whole segments and one cell more or less; velocities odd, a
# lone pair past a thread group's round, around the CTA sizes; ghosts and none
EDGES = [(1.5, 3, 5, 0), (2.0, 8, 31, 0), (3.0, 15, 64, 1), (4.0, 16, 129, 0), (1.2, 17, 33, 2), (6.0, 31, 256, 0),
         (2.5, 33, 18, 0), (1.8, 46, 255, 1), (5.0, 61, 128, 2), (3.5, 62, 49, 0)]


@pytest.mark.parametrize("coll", ["shakhov", "bgk"])
def test_fp32_segment_shapes_against_oracle(gpu_lib, coll):
    """Every shape, on a grid of CTAs per segment and a persistent one: within
    the FP32 split form's 1e-5 after 12 steps."""
    sets = KB.solver_sets([dict(KB.shock_config(Ma, nx, nu, coll=coll), nxg=ng) for Ma, nx, nu, ng in EDGES])
    refs = None
    for shape in [(8, 64), (16, 64), (16, 128), (16, 256), (32, 128), (32, 256)]:
        for persist in (0, 1):
            bt = KB.Batch(sets, "fp32")
            bt.set_tuning(*shape, persist)
            bt.init_initial()
            dt = bt.timestep()
            bt.step(12)
            outs = bt.download()
            bt.close()
            if refs is None:
                refs = []
                for KS, d in zip(sets, dt):
                    orc = oracle_for(KS)
                    orc.step(d, 12)
                    refs.append(orc.get_state())
            for k, (o, r) in enumerate(zip(outs, refs)):
                assert max(rho_u_t_error(o["prim"], r[1])) < 1e-5, (shape, persist, k)
                for key, x in (("h", r[2]), ("b", r[3])):
                    assert np.max(np.abs(o[key] - x)) < 1e-5 * np.max(np.abs(x)), (shape, persist, k, key)


LINES = [("three", sod(nx=3, nu=9)), ("four", shock(nx=4, nu=32)), ("ghosts", shock(nx=31, nu=33, ng=1)),
         ("widest", sod(nx=29, nu=255, coll="bgk")), ("wider", sod(nx=29, nu=257, coll="bgk")), ("long", sod(nx=157, nu=40))]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("name,cfg", LINES, ids=[c[0] for c in LINES])
def test_single_lines_against_oracle(gpu_lib, name, cfg, prec, tol):
    """35 steps: two graphs of 16 and single launches (segment kernels up to 256
    velocities, the general form beyond)."""
    KS, ctr, *faces, t = kitgpu.initialize(cfg, precision=prec)
    orc = oracle_for(KS)
    dt = kitgpu.timestep(KS, ctr, 0.0)
    kitgpu.step(KS, ctr, dt, 35)
    orc.step(dt, 35)
    got, ref = ctr.handle.download(), orc.get_state()
    assert max(rho_u_t_error(got["prim"], ref[1])) < tol
    for key, x in (("h", ref[2]), ("b", ref[3])):
        assert np.max(np.abs(got[key] - x)) < tol * np.max(np.abs(x)), key


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nsteps", [1, 64, 67])
def test_adaptive_lines_equal_single_steps(gpu_lib, prec, nsteps):
    """Time steps found on the device (chunks of 64) against one host
    timestep() per step: dt differs by rounding alone (FP64 on both sides), so
    the states agree to 1e-12 in FP64 and to FP32 rounding, 1e-5, in FP32."""
    cfg = sod(nx=50, nu=36)
    KS, a, *fa, t = kitgpu.initialize(cfg, precision=prec)
    KS, b, *fb, t = kitgpu.initialize(cfg, precision=prec)
    a.handle.step_cfl(KS.set.cfl, 0.0, 1e9, nsteps)
    for _ in range(nsteps):
        b.handle.step(b.handle.timestep(KS.set.cfl, 0.0, 1e9), 1)
    x, y = a.handle.download(), b.handle.download()
    tol = 1e-12 if prec == "fp64" else 1e-5
    assert max(rho_u_t_error(x["prim"], y["prim"])) < tol
    assert np.max(np.abs(x["h"] - y["h"])) < tol * np.max(y["h"])


@pytest.mark.parametrize("before", [1, 2, 5])
def test_pool_member_joins_after_any_number_of_steps(gpu_lib, before):
    """A solve that joins a pool after an odd or even number of steps starts in
    the buffer the next step reads: the state it has in a pool of its own, bit
    for bit (cells and velocities that an earlier member held are taken again)."""
    sets = KB.solver_sets([KB.shock_config(3.0, 61, 49), KB.shock_config(2.0, 40, 30), dict(KB.shock_config(4.0, 45, 33), nxg=1)])
    outs = []
    for alone in (False, True):
        pool = KB.Pool(sets[0], max_instances=4, max_cells=400)
        if not alone:
            first = [pool.add(KS)[0] for KS in sets[:2]]
            pool.step(before)
            pool.remove(first[1])
        slot = pool.add(sets[2])[0]
        pool.step(7)
        outs.append(pool.download(slot))
        pool.close()
    for k in ("w", "prim", "h", "b"):
        assert np.array_equal(outs[0][k], outs[1][k]), k
