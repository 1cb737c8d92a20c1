"""States to and from page-locked host arrays (read and written in place) and
pageable ones: rows of odd, padded and dense lengths, aligned to 16 bytes and
not, hold the same bits."""
import ctypes

import numpy as np
import pytest
import torch

import kitgpu
from kitgpu import _native as N
from cases import quadrant, sod

pytestmark = pytest.mark.gpu


def pinned(a, shift):
    """a copied to page-locked memory, its first element `shift` doubles past a
    16-byte boundary."""
    t = torch.empty(a.size + 2, dtype=torch.float64, pin_memory=True)
    assert t.data_ptr() % 16 == 0
    v = t[shift:shift + a.size].view(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("cfg", [quadrant(nx=7, ny=5, nu=13, nv=9), quadrant(nx=6, ny=9, nu=7, nv=6), sod(nx=41, nu=1 + 256),
                                 quadrant(nx=33, ny=31, nu=12, nv=12)], ids=["odd", "padded", "line", "dense"])
def test_page_locked_rows_hold_the_same_bits(gpu_lib, cfg, prec, shift):
    KS, ctr, *faces, t = kitgpu.initialize(cfg, precision=prec)
    h = ctr.handle
    rng = np.random.default_rng(4)
    s = h.download()
    state = [s["w"], s["prim"]] + [s[k] * rng.uniform(0.5, 1.5, s[k].shape) for k in ("h", "b")]
    h.upload(*state)
    want = h.download()
    p = [pinned(np.ascontiguousarray(x), shift) for x in state]
    h.init_equilibrium(*kitgpu.solver.initial_cells(KS))
    as_ptr = lambda x: ctypes.cast(x.data_ptr(), ctypes.POINTER(ctypes.c_double))
    h.call("kb_upload_state", *[as_ptr(x) for x in p])
    got = h.download()
    out = [pinned(np.zeros_like(x), shift) for x in state]
    h.call("kb_download_state", *[as_ptr(x) for x in out])
    for k, o in zip(("w", "prim", "h", "b"), out):
        assert np.array_equal(got[k], want[k]), k
        assert np.array_equal(o.numpy(), want[k]), k
