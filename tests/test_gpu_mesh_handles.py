"""Triangle-mesh solves side by side: handles of different velocity grids and
shapes stepped in turn, and shapes that change no result."""
import numpy as np
import pytest

from kitgpu import unstruct as US
from test_gpu_unstruct import _setup

pytestmark = pytest.mark.gpu


def _mesh(nv, coll, nx=6, ny=5):
    return _setup(dict(boundary="extra", collision=coll, nx=nx, ny=ny, nu=nv, nv=nv, jitter=0.2))[0]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("coll", ["bgk", "shakhov"])
def test_handles_of_large_and_small_grids_in_turn(gpu_lib, coll, prec):
    """A handle whose step needs much shared memory (64 x 64 velocities, and 32
    cells per CTA) beside one made later that needs little: each steps as it
    does alone, bit for bit."""
    big, wide, small = _mesh(64, coll, 4, 3), _mesh(18, coll), _mesh(5, coll)
    alone = []
    for KS, cb in ((big, 0), (wide, 32), (small, 1)):
        hd = US.init_fvm(KS, prec)
        if cb:
            hd.set_tuning(cb)
        dt = hd.timestep()
        r = [hd.step(dt, 1) for _ in range(4)]
        alone.append((dt, r, hd.download()))
        hd.close()
    hs = [US.init_fvm(KS, prec) for KS in (big, wide, small)]
    hs[1].set_tuning(32)
    hs[2].set_tuning(1)
    for k in range(4):
        for hd, (dt, r, _) in zip(hs, alone):
            assert np.array_equal(hd.step(dt, 1), r[k])
    for hd, (_, _, ref) in zip(hs, alone):
        got = hd.download()
        assert all(np.array_equal(got[k], ref[k]) for k in ("w", "prim", "h", "b"))
        hd.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,nv,coll", [(3, 3, 5, "bgk"), (5, 4, 9, "shakhov"), (13, 17, 11, "shakhov"),
                                           (20, 20, 16, "shakhov"), (12, 12, 12, "bgk"), (41, 37, 12, "bgk")])
def test_cells_per_cta_change_no_result(gpu_lib, nx, ny, nv, coll, prec):
    """The default and shapes given by hand: the same sums, bit for bit."""
    KS = _mesh(nv, coll, nx, ny)
    out = []
    for cb in (0, 1, 2, 3, 5, 8, 12, 32):
        hd = US.init_fvm(KS, prec)
        if cb:
            hd.set_tuning(cb)
        hd.step(hd.timestep(), 6)
        out.append(hd.download())
        hd.close()
    for o in out[1:]:
        assert all(np.array_equal(o[k], out[0][k]) for k in ("w", "prim", "h", "b"))
