"""Limits of the FP64 forms: exponentials far below the smallest number, fluxes
of the collision-dominated limit (dt many orders above tau), cold gases."""
import numpy as np
import pytest

import kitgpu
from kitgpu.solver import Handle, kb_config
from cases import oracle_for, quadrant, rho_u_t_error, sod
from test_gpu_f64 import call, lib  # noqa: F401 (the compiled forms)

pytestmark = pytest.mark.gpu


def test_exp2_tab_far_below_zero(lib):  # noqa: F811
    """0 for every product below 256 x -1022, around the 2^31 where its integer
    part leaves one word, the 2^51 where it leaves the mantissa, and at -inf;
    not a number for one that is none; 2^x on the last 256ths before zero."""
    near = [2.0 ** e + d for e in (18, 30, 31, 32, 33, 51, 52, 53, 62, 63, 64) for d in (-300.5, -1.0, 0.0, 1.0, 77.25)]
    x = -np.array([v for v in near if v > 1022 * 256] + [2.2e9, 3e9, 3.3e9, 5e9, 1e10, 1e12, 1e15, 1e16, 1e20, 1e100, 1e300, np.inf])
    assert np.all(call(lib, 2, x) == 0.0)
    a = np.linspace(1.0, 1e6, len(x))
    assert np.all(call(lib, 2, x / a * 1.5, a) == 0.0)
    rng = np.random.default_rng(7)
    x = -10.0 ** rng.uniform(6, 300, 2000)
    assert np.all(call(lib, 2, x) == 0.0)
    assert np.isnan(call(lib, 2, np.array([np.nan, -np.nan, -np.inf]), np.array([1.0, 1.0, 0.0]))).all()
    k = np.arange(1000 * 256, 1021 * 256, 37)
    assert np.array_equal(call(lib, 2, -256.0 * np.arange(0.0, 1022)), 2.0 ** -np.arange(0.0, 1022))
    got, want = call(lib, 2, -k.astype(float)), np.exp2(-k / 256.0)
    assert np.max(np.abs(got / want - 1.0)) < 8 * 2.0 ** -52


LIMITS = [("line", sod(nx=24, nu=25)), ("plane", quadrant(nx=10, ny=9, nu=13, nv=12))]


@pytest.mark.parametrize("Kn", [1e-9, 1e-11, 1e-13])
@pytest.mark.parametrize("flux", ["kcu", "ugks"])
@pytest.mark.parametrize("coll", ["bgk", "shakhov"])
@pytest.mark.parametrize("name,cfg", LIMITS, ids=[c[0] for c in LIMITS])
def test_collision_dominated_fluxes(gpu_lib, name, cfg, coll, flux, Kn):
    """FP64 KCU and UGKS with dt / tau from 10^6 to above 10^10, three steps."""
    KS, ctr, *faces, t = kitgpu.initialize(dict(cfg, flux=flux, collision=coll, knudsen=Kn))
    orc = oracle_for(KS)
    dt = kitgpu.timestep(KS, ctr, 0.0)
    kitgpu.step(KS, ctr, dt, 3)
    orc.step(dt, 3)
    got, ref = ctr.handle.download(), orc.get_state()
    assert max(rho_u_t_error(got["prim"], ref[1])) < 1e-12
    for key, x in (("h", ref[2]), ("b", ref[3])):
        assert np.max(np.abs(got[key] - x)) < 1e-12 * np.max(np.abs(x)), key


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("order", ["product", "shuffled"])
@pytest.mark.parametrize("dim", [1, 2])
def test_equilibrium_of_a_cold_gas(gpu_lib, dim, order, prec):
    """lambda up to 10^8, where lambda (u - U)^2 passes 2^31 / 369: no value above
    the exact one by more than rounding, none below zero."""
    KS = kitgpu.solver_set(sod(nx=9, nu=33) if dim == 1 else quadrant(nx=5, ny=4, nu=13, nv=10))
    vs = KS.vs
    u, w = (vs.u, vs.weights) if dim == 1 else (vs.flat(vs.u), vs.flat(vs.weights))
    v = None if dim == 1 else vs.flat(vs.v)
    perm = np.random.default_rng(1).permutation(len(u)) if order == "shuffled" else np.arange(len(u))
    h = Handle(kb_config(KS, prec), u[perm].copy(), None if dim == 1 else v[perm].copy(), w[perm].copy())
    lam = 10.0 ** np.linspace(0.0, 8.0, h.ncell)
    U = u[len(u) // 2 - 1] + 0.25 * (u[len(u) // 2] - u[len(u) // 2 - 1])
    P = np.stack([np.ones_like(lam), np.full_like(lam, U)] + ([np.zeros_like(lam)] if dim == 2 else []) + [lam], 1)
    h.init_equilibrium(P, P)
    got = h.download()
    x = lam[:, None] * ((u[perm][None] - U) ** 2 + (v[perm][None] ** 2 if dim == 2 else 0.0))
    H = (np.sqrt(lam / np.pi) if dim == 1 else lam / np.pi)[:, None] * np.exp(-x)
    # the exponent's rounding (2.5 x 2^-53), then a few more; FP32: its smallest number
    tol = (2.0 * (2.5 * np.minimum(x, 1100.0) + 8) * 2.0 ** -53 + (2.0 ** -23 if prec == "fp32" else 0.0)) * H
    tol += 1e-300 if prec == "fp64" else 2.0 ** -126 * (1 + KS.gas.K)
    for key, ref in (("h", H), ("b", H * KS.gas.K / (2.0 * lam[:, None]))):
        assert np.all(np.abs(got[key] - ref) <= tol), key
        assert np.all(got[key] >= 0.0), key
