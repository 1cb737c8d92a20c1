"""FP64 2D on product velocity grids: the Maxwellians' factors stand in the
staging buffer, a band of rows at a time, and take no memory of their own."""
import numpy as np
import pytest

from kitgpu.solver import Handle, initial_cells, kb_config, wall_states
import kitgpu
from cases import cavity, oracle_for, quadrant, rho_u_t_error

pytestmark = pytest.mark.gpu

# few velocities, whose factors outgrow the buffer: 2 bands and more, rows that
# bands do not divide, and one band
BANDS = [("kcu-shakhov-walls", cavity(nx=70, ny=101, nu=5, nv=4)), ("kcu-bgk-walls", cavity(nx=9, ny=131, nu=4, nv=5, coll="bgk")),
         ("ugks-bgk-extra", quadrant(nx=90, ny=83, nu=4, nv=3)), ("ugks-shakhov-extra", quadrant(nx=33, ny=64, nu=5, nv=5, coll="shakhov")),
         ("kfvs-shakhov-fix", quadrant(nx=40, ny=77, nu=3, nv=3, flux="kfvs", coll="shakhov", bc="fix", ng=0)),
         ("one-band", cavity(nx=12, ny=15, nu=13, nv=12)), ("three-rows", cavity(nx=20, ny=3, nu=4, nv=4))]


def _handle(KS, order):
    vs = KS.vs
    u, v, w = (vs.flat(x) for x in (vs.u, vs.v, vs.weights))
    h = Handle(kb_config(KS, "fp64"), u[order].copy(), v[order].copy(), w[order].copy())
    h.init_equilibrium(*initial_cells(KS))
    for side, prim in enumerate(wall_states(KS)):
        if KS.set.boundary[side] == "maxwell":
            h.set_wall(side, prim)
    return h


@pytest.mark.parametrize("name,cfg", BANDS, ids=[c[0] for c in BANDS])
def test_bands_against_exponentials_and_oracle(gpu_lib, name, cfg):
    """The same states as a velocity grid in another order, which is no product,
    and as the oracle, to the FP64 form's 1e-12 after 5 steps; the ordered grid
    holds no more device memory than the other (small solves: 8 MB)."""
    KS = kitgpu.solver_set(cfg)
    n = KS.vs.nu * KS.vs.nv
    perm = np.random.default_rng(4).permutation(n)
    a, b = _handle(KS, np.arange(n)), _handle(KS, perm)
    assert a.device_bytes() <= b.device_bytes() + (8 << 20)
    dt = a.timestep(KS.set.cfl, 0.0, 1e9)
    orc = oracle_for(KS)
    orc.step(dt, 5)
    a.step(dt, 5)
    b.step(dt, 5)
    x, y, ref = a.download(), b.download(), orc.get_state()
    back = np.argsort(perm)
    for s, o in ((x, np.arange(n)), (y, back)):
        assert max(rho_u_t_error(s["prim"], ref[1])) < 1e-12
        for key, r in (("h", ref[2]), ("b", ref[3])):
            assert np.max(np.abs(s[key][:, o] - r)) < 1e-12 * np.max(np.abs(r)), key


def test_product_grids_take_no_more_memory(gpu_lib):
    """A grid whose staging buffer is large: exactly as much as in another order."""
    KS = kitgpu.solver_set(cavity(nx=40, ny=40, nu=24, nv=24))
    n = KS.vs.nu * KS.vs.nv
    a, b = _handle(KS, np.arange(n)), _handle(KS, np.random.default_rng(4).permutation(n))
    assert a.device_bytes() == b.device_bytes()


def test_factors_and_uploads_share_the_buffer(gpu_lib):
    """Steps between uploads and downloads of pageable arrays, which cross the
    same buffer: a state uploaded again steps on as it did."""
    KS = kitgpu.solver_set(cavity(nx=30, ny=41, nu=5, nv=5))
    a = _handle(KS, np.arange(25))
    dt = a.timestep(KS.set.cfl, 0.0, 1e9)
    a.step(dt, 3)
    s = a.download()
    a.step(dt, 4)
    first = a.download()
    a.upload(s["w"], s["prim"], s["h"], s["b"])
    a.step(dt, 4)
    again = a.download()
    for k in ("w", "prim", "h", "b"):
        assert np.array_equal(first[k], again[k]), k
