"""The default shape of the triangle-mesh step (cells per CTA, and in FP64 the
parts of a cell that warps take) on meshes and velocity grids of several sizes,
against a shape given by hand."""
import numpy as np
import pytest

from kitgpu import unstruct as US
from test_gpu_unstruct import _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-13), ("fp32", 0.0)])
@pytest.mark.parametrize("nx,ny,nv,coll", [(3, 3, 5, "bgk"), (5, 4, 9, "shakhov"), (13, 17, 11, "shakhov"), (41, 37, 12, "bgk")])
def test_default_shape_equals_a_given_one(gpu_lib, nx, ny, nv, coll, prec, tol):
    """FP32: the same sums, bit for bit.  FP64: a cell's sums may be formed in
    two parts, a rounding apart (2^-53 of the sums a step, 6 steps, a condition
    below 100: 1e-13)."""
    KS, orc = _setup(dict(boundary="extra", collision=coll, nx=nx, ny=ny, nu=nv, nv=nv, jitter=0.2))
    out = []
    for cb in (0, 5):
        hd = US.init_fvm(KS, prec)
        if cb:
            hd.set_tuning(cb)
        hd.step(hd.timestep(), 6)
        out.append(hd.download())
        hd.close()
    for k in ("w", "prim", "h", "b"):
        assert np.max(np.abs(out[0][k] - out[1][k])) <= tol * np.max(np.abs(out[1][k])), k


@pytest.mark.parametrize("coll,nv,cb", [("bgk", 9, 0), ("shakhov", 12, 0), ("shakhov", 16, 32), ("bgk", 5, 1)])
def test_factored_maxwellians_equal_exponentials(gpu_lib, coll, nv, cb):
    """FP64: a velocity grid in another order is no product, so its relaxation
    takes the exponentials where the ordered one takes products of factors: the
    same states to the FP64 form's 1e-12 after 6 steps."""
    out = []
    for shuffle in (False, True):
        KS, orc = _setup(dict(boundary="extra", collision=coll, nx=7, ny=6, nu=nv, nv=nv, jitter=0.2))
        vs = KS.vs
        n = vs.u.size
        perm = np.random.default_rng(3).permutation(n) if shuffle else np.arange(n)
        for k in ("u", "v", "weights"):
            a = getattr(vs, k)
            setattr(vs, k, a.ravel(order="F")[perm].reshape(a.shape, order="F"))
        hd = US.init_fvm(KS, "fp64")
        if cb:
            hd.set_tuning(cb)
        hd.step(hd.timestep(), 6)
        s = hd.download()
        hd.close()
        back = np.argsort(perm)
        out.append((s["w"], s["prim"], s["h"][:, back], s["b"][:, back]))
    for x, y in zip(*out):
        assert np.max(np.abs(x - y)) < 1e-12 * np.max(np.abs(y))


@pytest.mark.parametrize("n", [44, 65])
def test_residual_of_many_ctas(gpu_lib, n):
    """One cell per CTA on meshes on either side of the 2,048 CTAs whose sums one
    CTA adds by itself: the residual of 8 cells per CTA, to the rounding of a
    sum of at most 10^4 terms of one sign (1e-11)."""
    KS, orc = _setup(dict(boundary="extra", collision="bgk", nx=n // 2, ny=n, nu=5, nv=5, jitter=0.2))
    res = []
    for cb in (1, 8):
        hd = US.init_fvm(KS, "fp64")
        hd.set_tuning(cb)
        res.append(np.array(hd.step(hd.timestep(), 3)))
        hd.close()
    assert np.all(np.abs(res[0] - res[1]) <= 1e-11 * np.abs(res[1])), res
