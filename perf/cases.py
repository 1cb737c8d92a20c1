"""The work that programs on this framework have it do, as cases to be measured.

Every case is one whole use of a public entry point on a solver that the
program keeps: start (or restart) a solve, advance it by a run of time steps,
take the solution.  The kinds:

  line      one 1D2F1V solve (Handle.init_equilibrium, timestep, step, download)
  adaptive  the same with the time step renewed before every step (step_cfl)
  plane     one 2D2F2V solve, from a macroscopic state
  restart   one 2D2F2V solve continued from a checkpoint's w, prim, h, b
  shocks    an ensemble of 1D shock structures advanced together (Batch)
  mesh      a solve on a triangle mesh (UnstructHandle)
  serve     a burst of small requests through the serving loop (Server.run)

The plain form ("f64") returns FP64 arrays; the FP32-split form ("f32") keeps
h and b in FP32 on the device, and its results are returned in FP32.
Library defaults everywhere: no autotuning, as in initialize() and solve().

exact() restates one pass in 64 bits with plain torch operations.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "kitbase.jl_gb300"))

PI = math.pi


# ------------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call in use: a coarse Sod tube with the per-step dt option,
        # where every step waits for the device's CFL reduction
        dict(name="sod_64x33_f64_adaptive", kind="adaptive", nx=64, nu=33, flux="kfvs", coll="bgk",
             prec="f64", steps=16),
        # the Sod tube of the tests and the benchmark, solved to t = 0.2: 504 short steps
        dict(name="sod_200x101_f32", kind="line", nx=200, nu=101, flux="kfvs", coll="shakhov",
             prec="f32", steps=504),
        # the lid-driven cavity of the tests and the benchmark, plain FP64 form
        dict(name="cavity_64x28_f64", kind="plane", nx=64, ny=64, nu=28, nv=28, flux="kcu",
             coll="shakhov", bc="maxwell", prec="f64", steps=40, full=True),
        # the same cavity in the FP32-split form: a chunk of its 2000 steps
        dict(name="cavity_64x28_f32", kind="plane", nx=64, ny=64, nu=28, nv=28, flux="kcu",
             coll="shakhov", bc="maxwell", prec="f32", steps=200, full=False),
        # the benchmark's headline: four-quadrant Riemann problem, 1.07e9 cell-velocity points
        dict(name="quadrant_512x64_f32", kind="plane", nx=512, ny=512, nu=64, nv=64, flux="ugks",
             coll="bgk", bc="extra", prec="f32", steps=10, full=False),
        # the same physics in the plain FP64 form at a size that form is run at
        dict(name="quadrant_128x32_f64", kind="plane", nx=128, ny=128, nu=32, nv=32, flux="ugks",
             coll="bgk", bc="extra", prec="f64", steps=6, full=False),
        # ragged sizes (rows of 1073 velocities: padded), second flux and collision model,
        # continued from a checkpoint in page-locked memory and checkpointed again
        dict(name="restart_131x97_f32", kind="restart", nx=131, ny=97, nu=37, nv=29, flux="kfvs",
             coll="shakhov", bc="fix", prec="f32", steps=40),
        # 512 ragged shock structures (50..400 cells, 48..200 velocities) in one batch
        dict(name="shocks_512_f32", kind="shocks", n=512, mix=20261203, coll="shakhov", prec="f32",
             steps=200),
        # a small ensemble in the plain FP64 form
        dict(name="shocks_24_f64", kind="shocks", n=24, mix=7, coll="shakhov", prec="f64", steps=40),
        # the benchmark's triangle mesh: 294,912 triangles, 16 x 16 velocities
        dict(name="mesh_384_f32", kind="mesh", n=384, nu=16, nv=16, coll="bgk", prec="f32", steps=20,
             full=False),
        # a mesh of the size of the tests' gmsh files, Shakhov, FP64, state in and out
        dict(name="mesh_20_f64", kind="mesh", n=20, nu=16, nv=16, coll="shakhov", prec="f64", steps=60,
             full=True),
        # a burst of the served mix: Sod tubes share a pool, small cavities a group
        dict(name="serve_14_f32", kind="serve", lines=8, planes=6, mix=5, prec="f32", steps=100),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["adaptive", "line", "plane", "plane", "plane", "restart", "shocks", "mesh", "serve"])
    if kind in ("adaptive", "line"):
        c = dict(kind=kind, nx=_log(rng, 64, 2048), nu=rng.randint(32, 256),
                 flux=rng.choice(["kfvs", "kfvs", "kcu", "ugks"]), coll=rng.choice(["bgk", "shakhov"]),
                 prec=rng.choice(["f64", "f32"]))
        c["steps"] = rng.randint(8, 32) if kind == "adaptive" else rng.randint(64, 256)
        return c
    if kind in ("plane", "restart"):
        prec = rng.choice(["f32", "f32", "f64"])
        form = rng.choice(["cavity", "quadrant", "kfvs"]) if kind == "plane" else "kfvs"
        if form == "cavity":
            n, v = (16, 128), (16, 48)
        elif form == "quadrant":
            n, v = (64, 400), (16, 64)
        else:
            n, v = (48, 160), (16, 40)
        if prec == "f64":
            n, v = (16, 96), (12, 32)
        c = dict(kind=kind, nx=_log(rng, *n), ny=_log(rng, *n), nu=rng.randint(*v), nv=rng.randint(*v), prec=prec)
        if form == "cavity":
            c.update(flux=rng.choice(["kcu", "ugks"]), coll="shakhov", bc="maxwell")
        elif form == "quadrant":
            c.update(flux="ugks", coll="bgk", bc="extra")
        else:
            c.update(flux="kfvs", coll="shakhov", bc="fix")
        cv = c["nx"] * c["ny"] * c["nu"] * c["nv"]
        c["steps"] = max(2, min(64, int((3e9 if prec == "f32" else 6e7) / cv)))
        if kind == "plane":
            c["full"] = cv < 4e6
        return c
    if kind == "shocks":
        prec = rng.choice(["f32", "f32", "f64"])
        n = _log(rng, 8, 512) if prec == "f32" else _log(rng, 4, 48)
        return dict(kind=kind, n=n, mix=rng.randint(1, 1 << 20), coll=rng.choice(["bgk", "shakhov"]), prec=prec,
                    steps=rng.randint(20, 100) if prec == "f32" else rng.randint(8, 40))
    if kind == "mesh":
        prec = rng.choice(["f32", "f32", "f64"])
        n = _log(rng, 16, 320) if prec == "f32" else _log(rng, 12, 80)
        return dict(kind=kind, n=n, nu=rng.randint(12, 20), nv=rng.randint(12, 20), coll=rng.choice(["bgk", "shakhov"]),
                    prec=prec, steps=rng.randint(8, 20), full=n < 40)
    return dict(kind="serve", lines=rng.randint(2, 10), planes=rng.randint(1, 6), mix=rng.randint(1, 1 << 20), prec="f32",
                steps=20 * rng.randint(2, 5))


# ------------------------------------------------------------ configurations

def _cfg_line(c):
    return dict(matter="gas", case="sod", space="1d2f1v", flux=c["flux"], collision=c["coll"], nSpecies=1,
                interpOrder=2, limiter="vanleer", boundary="fix", cfl=0.5, maxTime=1e9, x0=0.0, x1=1.0,
                nx=c["nx"], nxg=0, umin=-5.0, umax=5.0, nu=c["nu"], vMeshType="newton", knudsen=1e-4, mach=0.0,
                prandtl=2.0 / 3.0, inK=2.0, omega=0.81, alphaRef=1.0, omegaRef=0.5)


def _cfg_plane(c):
    wall, ghost = c["bc"] == "maxwell", 1 if c["bc"] == "extra" else 0
    lim = 5.0 if wall else 6.0
    return dict(matter="gas", case="cavity" if wall else "quadrant", space="2d2f2v", flux=c["flux"],
                collision=c["coll"], nSpecies=1, interpOrder=2, limiter="vanleer", boundary=c["bc"],
                cfl=0.8 if wall else 0.5, maxTime=1e9, x0=0.0, x1=1.0, nx=c["nx"], nxg=ghost, y0=0.0, y1=1.0,
                ny=c["ny"], nyg=ghost, umin=-lim, umax=lim, nu=c["nu"], vmin=-lim, vmax=lim, nv=c["nv"],
                vMeshType="newton", knudsen=0.075 if wall else 1e-3, mach=0.0, prandtl=2.0 / 3.0, inK=1.0,
                omega=0.72 if wall else 0.81, alphaRef=1.0, omegaRef=0.5, uLid=0.15, vLid=0.0, tLid=1.0)


def _cfg_shocks(c, seed):
    """The ensemble's configurations: sizes from the case, Mach numbers from the seed."""
    size, mach = np.random.default_rng(c["mix"]), np.random.default_rng(seed)
    out = []
    for _ in range(c["n"]):
        nx, nu, ma = int(size.integers(50, 401)), int(size.integers(48, 201)), float(mach.uniform(1.2, 8.0))
        lim = 5.0 + 2.0 * ma
        out.append(dict(matter="gas", case="shock", space="1d2f1v", flux="kfvs", collision=c["coll"], nSpecies=1,
                        interpOrder=2, limiter="vanleer", boundary="fix", cfl=0.5, maxTime=1e9, x0=-35.0, x1=35.0,
                        nx=nx, nxg=0, umin=-lim, umax=lim, nu=nu, vMeshType="rectangle", knudsen=1.0, mach=ma,
                        prandtl=2.0 / 3.0, inK=2.0, omega=0.72, alphaRef=1.0, omegaRef=0.5))
    return out


def _cfg_serve(c, seed):
    """The burst's configurations: sizes from the case, Knudsen numbers from the seed."""
    size, kn = np.random.default_rng(c["mix"]), np.random.default_rng(seed)
    lines, planes = [], []
    for _ in range(c["lines"]):
        nx, nu = int(round(math.exp(size.uniform(math.log(64), math.log(2048))))), int(size.integers(32, 257))
        lines.append(dict(_cfg_line(dict(nx=nx, nu=nu, flux="kfvs", coll="shakhov")),
                          knudsen=math.exp(kn.uniform(math.log(1e-4), math.log(1e-2)))))
    for _ in range(c["planes"]):
        n, v = int(round(math.exp(size.uniform(math.log(16), math.log(96))))), int(size.integers(16, 41))
        while (n - 0.5) * (1.0 / n) + 0.5 * (1.0 / n) != 1.0:  # the lid's state holds where y == y1 exactly
            n += 1
        planes.append(dict(_cfg_plane(dict(nx=n, ny=n, nu=v, nv=v, flux="kcu", coll="shakhov", bc="maxwell")),
                           knudsen=math.exp(kn.uniform(math.log(1e-3), math.log(1.0)))))
    return lines, planes


# ------------------------------------------------------------- initial states

def _cons(p, gamma):
    """Conserved variables of primitive ones [rho, U, (V,) lambda] (last axis)."""
    r, l = p[..., 0], p[..., -1]
    m = [r * p[..., k] for k in range(1, p.shape[-1] - 1)]
    e = 0.5 * r / l / (gamma - 1.0) + 0.5 * sum(x * p[..., k + 1] for k, x in enumerate(m))
    stack = np.stack if isinstance(p, np.ndarray) else torch.stack
    return stack([r] + m + [e], -1)


def _gamma(inK, dim):
    return (inK + 3.0) / (inK + 1.0) if dim == 1 else (inK + 4.0) / (inK + 2.0)


def _line_prim(cfg, seed):
    """A Sod tube whose two states vary with the seed; cells of [0, 1], no ghosts."""
    r = np.random.default_rng(seed)
    left = np.array([r.uniform(0.9, 1.1), r.uniform(-0.1, 0.1), r.uniform(0.45, 0.55)])
    right = np.array([r.uniform(0.11, 0.14), r.uniform(-0.1, 0.1), r.uniform(0.58, 0.68)])
    x = (np.arange(cfg["nx"]) + 0.5) / cfg["nx"]
    return np.where((x <= 0.5)[:, None], left, right)


def _plane_prim(cfg, seed):
    """Macroscopic state over all cells incl. ghosts, [ny + 2g, nx + 2g, 4]: four
    quadrants, or for a cavity a gas at rest with smooth disturbances."""
    r = np.random.default_rng(seed)
    nx, ny, g = cfg["nx"], cfg["ny"], cfg["nxg"]
    x = (np.arange(-g, nx + g) + 0.5)[None, :] / nx + np.zeros((ny + 2 * g, 1))
    y = (np.arange(-g, ny + g) + 0.5)[:, None] / ny + np.zeros((1, nx + 2 * g))
    if cfg["case"] == "cavity":
        ph = r.uniform(0, 2 * PI, (4, 2))
        a = r.uniform(0.5, 1.0, 4) * np.array([0.05, 0.05, 0.05, 0.05])
        f = [a[k] * np.cos(2 * PI * x + ph[k, 0]) * np.cos(2 * PI * y + ph[k, 1]) for k in range(4)]
        return np.stack([1.0 + f[0], f[1], f[2], 1.0 + f[3]], -1)
    q = np.stack([r.uniform(0.1, 1.5, 4), r.uniform(-0.5, 0.5, 4), r.uniform(-0.5, 0.5, 4), r.uniform(0.4, 1.2, 4)], -1)
    return q[np.where(x > 0.5, np.where(y > 0.5, 0, 3), np.where(y > 0.5, 1, 2))]


def _walls(cfg):
    """Wall states of the four sides, one per face: at rest, the lid on top moving."""
    rest, lid = [1.0, 0.0, 0.0, 1.0], [1.0, cfg["uLid"], cfg["vLid"], cfg["tLid"]]
    return [np.tile(rest, (cfg["ny"], 1)), np.tile(rest, (cfg["ny"], 1)), np.tile(rest, (cfg["nx"], 1)),
            np.tile(lid, (cfg["nx"], 1))]


def _shock_prims(cfgs):
    """Rankine-Hugoniot states on both sides of the middle, upstream [1, U, 0.5]."""
    out = []
    for c in cfgs:
        g, ma, lam = _gamma(c["inK"], 1), c["mach"], 0.5
        mr = math.sqrt((ma ** 2 * (g - 1) + 2) / (2 * g * ma ** 2 - (g - 1)))
        rt = (1 + (g - 1) / 2 * ma ** 2) * (2 * g / (g - 1) * ma ** 2 - 1) / (ma ** 2 * (2 * g / (g - 1) + (g - 1) / 2))
        s = math.sqrt(g / (2 * lam))
        left = np.array([1.0, ma * s, lam])
        right = np.array([(g + 1) * ma ** 2 / ((g - 1) * ma ** 2 + 2), mr * s * math.sqrt(rt), lam / rt])
        x = np.arange(c["nx"]) + 0.5 <= 0.5 * c["nx"]
        out.append(np.where(x[:, None], left, right))
    return out


def _kick(h, seed):
    """h away from equilibrium, as a checkpoint from the middle of a solve holds it."""
    n = torch.arange(h.shape[-1], dtype=torch.float64, device=h.device)
    m = torch.arange(h.shape[0], dtype=torch.float64, device=h.device)
    r = random.Random(seed)
    a, b, c = r.uniform(0.02, 0.06), r.uniform(0.01, 0.03), r.uniform(0, 6)
    return h * (1.0 + a * torch.cos(0.37 * n + c)[None, :] * torch.cos(b * m)[:, None])


def _restart_state(cfg, c, seed, dev):
    """w, prim [ncell, 4] and h, b [ncell, nu nv] of a solve under way, on the device."""
    p = torch.from_numpy(_plane_prim(cfg, seed).reshape(-1, 4)).to(dev)
    u, v, _ = _grid2(cfg, dev)
    h = _maxwell(p[:, None, :], u, v)
    b = h * cfg["inK"] / (2.0 * p[:, None, 3])
    return _cons(p, _gamma(cfg["inK"], 2)), p, _kick(h, seed), _kick(b, seed + 1)


def _mesh_points(c):
    """The unit square in n x n quads with moved inner points, each quad cut along
    alternating diagonals."""
    n = c["n"]
    r = np.random.default_rng(7)
    s = np.linspace(0.0, 1.0, n + 1)
    P = np.stack(np.meshgrid(s, s), -1)
    P[1:-1, 1:-1] += r.uniform(-1, 1, (n - 1, n - 1, 2)) * (0.2 / n)
    j, i = np.divmod(np.arange(n * n), n)
    a = j * (n + 1) + i
    b, d, e = a + 1, a + n + 1, a + n + 2
    even = ((i + j) % 2 == 0)[:, None]
    first = np.where(even, np.stack([a, b, e], -1), np.stack([a, b, d], -1))
    second = np.where(even, np.stack([a, e, d], -1), np.stack([b, e, d], -1))
    return P.reshape(-1, 2), np.stack([first, second], 1).reshape(-1, 3)


_MESH_KEPT = {}


def _mesh(c):
    """The mesh tables (they depend on the case alone; the last one is kept)."""
    from kitgpu import unstruct
    if c["n"] not in _MESH_KEPT:
        _MESH_KEPT.clear()
        _MESH_KEPT[c["n"]] = unstruct.build_mesh(*_mesh_points(c), boundary="extra")
    return _MESH_KEPT[c["n"]]


def _mesh_state(center, c, seed, dev):
    r = np.random.default_rng(seed)
    x, y = (torch.from_numpy(np.ascontiguousarray(center[:, k])).to(dev) for k in (0, 1))
    f = [float(r.uniform(0.1, 0.3)) * torch.cos(2 * PI * x + float(r.uniform(0, 6))) * torch.cos(2 * PI * y + float(r.uniform(0, 6)))
         for _ in range(4)]
    p = torch.stack([1 + f[0], f[1], f[2], 1 + f[3]], -1)
    u, v, _ = _grid2(dict(umin=-5.0, umax=5.0, nu=c["nu"], vmin=-5.0, vmax=5.0, nv=c["nv"], vMeshType="rectangle"), dev)
    h = _maxwell(p[:, None, :], u, v)
    return _cons(p, _gamma(1.0, 2)), p, h, h * 1.0 / (2.0 * p[:, None, 3])


# ------------------------------------------------------------------ one pass

def _pinned(x):
    y = torch.empty(x.shape, dtype=torch.float64, pin_memory=True)
    y.copy_(x)
    return y


def _ptr(x):
    return ctypes.cast(x.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _prec(c):
    return {"f64": "fp64", "f32": "fp32"}[c["prec"]]


def prepare(case, seed):
    import kitgpu
    from kitgpu.solver import Handle, kb_config
    k = case["kind"]
    s = dict(case=case)
    if k in ("adaptive", "line"):
        cfg = _cfg_line(case)
        KS = kitgpu.solver_set(cfg)
        s["handle"] = Handle(kb_config(KS, _prec(case)), KS.vs.u, None, KS.vs.weights)
        s["prim"] = _line_prim(cfg, seed)
        s["w"] = _cons(s["prim"], KS.gas.gamma)
    elif k in ("plane", "restart"):
        cfg = _cfg_plane(case)
        KS = kitgpu.solver_set(cfg)
        vs = KS.vs
        hd = s["handle"] = Handle(kb_config(KS, _prec(case)), vs.flat(vs.u), vs.flat(vs.v), vs.flat(vs.weights))
        if case["bc"] == "maxwell":
            for side, p in enumerate(_walls(cfg)):
                hd.set_wall(side, p)
        if k == "plane":
            s["prim"] = _plane_prim(cfg, seed).reshape(-1, 4)
            s["w"] = _cons(s["prim"], KS.gas.gamma)
        else:
            s["state"] = [_pinned(x) for x in _restart_state(cfg, case, seed, "cuda")]
        if case.get("full", True):
            n = (hd.ncell, hd.nvel)
            s["out"] = [torch.empty(q, dtype=torch.float64, pin_memory=True) for q in ((n[0], 4), (n[0], 4), n, n)]
    elif k == "shocks":
        from kitgpu.batch import Batch
        cfgs = _cfg_shocks(case, seed)
        s["batch"] = Batch([kitgpu.solver_set(c, lamL=0.5) for c in cfgs], _prec(case))
        p = _shock_prims(cfgs)
        s["prim"] = np.ascontiguousarray(np.concatenate(p))
        s["w"] = _cons(s["prim"], _gamma(2.0, 1))
    elif k == "mesh":
        from kitgpu import unstruct
        m = _mesh(case)
        KS = unstruct.unstruct_solver_set(m, nu=case["nu"], nv=case["nv"], Kn=0.075, Pr=2.0 / 3.0, collision=case["coll"],
                                          cfl=0.5, maxTime=1e9)
        s["handle"] = unstruct.UnstructHandle(KS, _prec(case))
        state = [x.cpu().numpy() for x in _mesh_state(m.cell_center, case, seed, "cuda")]
        s["handle"].upload(*state)
        s["dt"] = s["handle"].timestep()
        if case["full"]:
            s["state"] = state
        else:
            s["out"] = [torch.empty((m.ncell, 4), dtype=torch.float64, pin_memory=True) for _ in range(2)]
    else:
        s["requests"] = _cfg_serve(case, seed)
    kitgpu.load()
    return s


def _given(case, x):
    """A result in the precision of the form that was asked for."""
    x = torch.from_numpy(x) if isinstance(x, np.ndarray) else x
    return x.float() if case["prec"] == "f32" else x


def run(state):
    case = state["case"]
    k, n = case["kind"], case["steps"]
    if k == "serve":
        from kitgpu.serve import Request, Server
        lines, planes = state["requests"]
        reqs = [Request(i, 0.0, cfg, n, 0.0) for i, cfg in enumerate(lines + planes)]
        Server(precision="fp32", hbm_budget=8 << 30, max_slots=32).run(reqs, keep_results=True)
        return {"prim": [_given(case, r.result["prim"]) for r in reqs], "w": [_given(case, r.result["w"]) for r in reqs]}
    if k == "shocks":
        from kitgpu import _native as N
        b = state["batch"]
        N.check(b.lib.kb_batch_init_equilibrium(b.h, N.ptr(state["w"]), N.ptr(state["prim"])))
        b.timestep()
        b.step(n)
        w, p = np.empty_like(state["w"]), np.empty_like(state["prim"])
        N.check(b.lib.kb_batch_download(b.h, N.ptr(w), N.ptr(p), None, None))
        return {"w": _given(case, w), "prim": _given(case, p)}
    hd = state["handle"]
    if k == "mesh":
        if case["full"]:
            hd.upload(*state["state"])
            hd.step(state["dt"], n)
            return {q: _given(case, x) for q, x in hd.download().items()}
        from kitgpu import _native as N
        hd.step(state["dt"], n)
        w, p = state["out"]
        N.check(hd.lib.kb_us_download(hd.h, _ptr(w), _ptr(p), None, None))
        return {"w": _given(case, w), "prim": _given(case, p)}
    if k == "restart":
        hd.call("kb_upload_state", *[_ptr(x) for x in state["state"]])
    else:
        hd.init_equilibrium(state["w"], state["prim"])
    cfl = 0.8 if case.get("bc") == "maxwell" else 0.5
    if k == "adaptive":
        hd.step_cfl(cfl, 0.0, 1e9, n)
    else:
        hd.step(hd.timestep(cfl, 0.0, 1e9), n)
    if "out" in state:
        hd.call("kb_download_state", *[_ptr(x) for x in state["out"]])
        return {q: _given(case, x) for q, x in zip(("w", "prim", "h", "b"), state["out"])}
    want = ("w", "prim", "h", "b") if k in ("line", "adaptive") else ("w", "prim")
    return {q: _given(case, x) for q, x in hd.download(want).items()}


# ------------------------------------------------------------------- its work

def _points(case):
    """Cell-velocity points advanced by one step."""
    k = case["kind"]
    if k in ("adaptive", "line"):
        return case["nx"] * case["nu"]
    if k in ("plane", "restart"):
        return case["nx"] * case["ny"] * case["nu"] * case["nv"]
    if k == "shocks":
        return sum(c["nx"] * c["nu"] for c in _cfg_shocks(case, 0))
    if k == "mesh":
        return 2 * case["n"] ** 2 * case["nu"] * case["nv"]
    lines, planes = _cfg_serve(case, 0)
    return sum(c["nx"] * c["nu"] for c in lines) + sum(c["nx"] * c["ny"] * c["nu"] * c["nv"] for c in planes)


def work(case):
    """A step reads h and b once and writes them once, at 8 or 4 bytes; a restart
    also moves the FP64 state in and out.  Operations per point: slopes, fluxes and
    their moments, the equilibrium and the relaxation, as the formulas count them."""
    n, size = _points(case), 8 if case["prec"] == "f64" else 4
    per = {"kfvs": 90, "kcu": 130, "ugks": 220}[case.get("flux", "kfvs")]
    if case["kind"] in ("plane", "restart", "serve"):
        per *= 1.8
    b = 4.0 * size * n * case["steps"]
    if case["kind"] == "restart":
        b += 32.0 * n
    return {"bytes": b, "flops": float(per) * n * case["steps"]}


# ------------------------------------------------- the same pass in 64 bits

def _cotes(n):
    c = np.array([14 / 45 if i in (1, n) else 28 / 45 if (i - 5) % 4 == 0 else 24 / 45 if (i - 3) % 4 == 0 else 64 / 45
                  for i in range(1, n + 1)])
    return c


def _grid1(cfg, kind="u"):
    lo, hi, n = cfg[kind + "min"], cfg[kind + "max"], cfg["n" + kind]
    d = (hi - lo) / n
    return lo + (np.arange(n) + 0.5) * d, (_cotes(n) if cfg["vMeshType"] == "newton" else np.ones(n)) * d


def _grid2(cfg, dev):
    (u, wu), (v, wv) = _grid1(cfg, "u"), _grid1(cfg, "v")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a.ravel())).to(dev)  # u fastest
    one = np.ones((cfg["nv"], cfg["nu"]))
    return t(one * u[None, :]), t(one * v[:, None]), t(wv[:, None] * wu[None, :])


def _maxwell(p, u, v=None):
    l = p[..., -1]
    if v is None:
        return p[..., 0] * torch.sqrt(l / PI) * torch.exp(-l * (u - p[..., 1]) ** 2)
    return p[..., 0] * (l / PI) * torch.exp(-l * ((u - p[..., 1]) ** 2 + (v - p[..., 2]) ** 2))


def _prims(w, gamma):
    r, e = w[..., 0], w[..., -1]
    m = [w[..., k] for k in range(1, w.shape[-1] - 1)]
    return torch.stack([r] + [x / r for x in m] + [0.5 * r / (gamma - 1) / (e - 0.5 * sum(x * x for x in m) / r)], -1)


def _limited(q, d, ends):
    """van Leer slopes along axis 1 of the cells q; one-sided or zero at the ends."""
    g = (q[:, 1:] - q[:, :-1]) / d
    a, b = g[:, :-1], g[:, 1:]
    s = torch.zeros_like(q)
    s[:, 1:-1] = (torch.sign(a) + torch.sign(b)) * a.abs() * b.abs() / (a.abs() + b.abs() + 1e-7)
    if ends:
        s[:, 0], s[:, -1] = g[:, 0], g[:, -1]
    return s


class _Gas:
    def __init__(self, cfg, dim):
        self.K, self.Pr, self.om, self.D = cfg["inK"], cfg["prandtl"], cfg["omega"], dim
        self.gamma = _gamma(cfg["inK"], dim)
        a, o = cfg["alphaRef"], cfg["omegaRef"]
        self.mu = 5.0 * (a + 1) * (a + 2) * math.sqrt(PI) / (4 * a * (5 - 2 * o) * (7 - 2 * o)) * cfg["knudsen"]

    def tau(self, p):
        return self.mu * 2.0 * p[..., -1] ** (1.0 - self.om) / p[..., 0]


def _gauss(p, K):
    """Half- and full-range moments of the unit Maxwellian of each state."""
    l, U = p[..., -1], p[..., 1]
    sq, e = torch.sqrt(l), torch.exp(-l * U * U) / torch.sqrt(PI * l) * 0.5
    L, R = [0.5 * torch.erfc(-sq * U)], [0.5 * torch.erfc(sq * U)]
    L.append(U * L[0] + e)
    R.append(U * R[0] - e)
    V = None
    if p.shape[-1] == 4:
        V = [torch.ones_like(l), p[..., 2]]
    for i in range(2, 7):
        for M, X in ((L, U), (R, U)) + (((V, p[..., 2]),) if V else ()):
            M.append(X * M[i - 1] + 0.5 * (i - 1) * M[i - 2] / l)
    xi = [torch.ones_like(l), 0.5 * K / l, (K * K + 2 * K) / (4 * l * l)]
    return L, R, [a + b for a, b in zip(L, R)], V, xi


def _mc(M, V, xi, a, b, d):
    """Conserved moments of u^a v^b xi^d."""
    x, y = xi[d // 2], xi[(d + 2) // 2]
    if V is None:
        return torch.stack([M[a] * x, M[a + 1] * x, 0.5 * (M[a + 2] * x + M[a] * y)], -1)
    return torch.stack([M[a] * V[b] * x, M[a + 1] * V[b] * x, M[a] * V[b + 1] * x,
                        0.5 * (M[a + 2] * V[b] * x + M[a] * V[b + 2] * x + M[a] * V[b] * y)], -1)


def _mcs(s, M, V, xi, a):
    """Conserved moments of u^a (s . psi)."""
    c = lambda k: s[..., k:k + 1]
    if V is None:
        return c(0) * _mc(M, V, xi, a, 0, 0) + c(1) * _mc(M, V, xi, a + 1, 0, 0) + 0.5 * c(2) * (
            _mc(M, V, xi, a + 2, 0, 0) + _mc(M, V, xi, a, 0, 2))
    return (c(0) * _mc(M, V, xi, a, 0, 0) + c(1) * _mc(M, V, xi, a + 1, 0, 0) + c(2) * _mc(M, V, xi, a, 1, 0)
            + 0.5 * c(3) * (_mc(M, V, xi, a + 2, 0, 0) + _mc(M, V, xi, a, 2, 0) + _mc(M, V, xi, a, 0, 2)))


def _pdf_slope(p, s, K):
    D = p.shape[-1] - 2
    r, l = p[..., 0], p[..., -1]
    U = [p[..., k] for k in range(1, D + 1)]
    c2 = sum(x * x for x in U)
    last = 4 * l * l / (K + D) / r * (2 * s[..., -1] - sum(2 * x * s[..., k + 1] for k, x in enumerate(U))
                                      + s[..., 0] * (c2 - 0.5 * (K + D) / l))
    mid = [2 * l / r * (s[..., k + 1] - x * s[..., 0]) - x * last for k, x in enumerate(U)]
    first = s[..., 0] / r - sum(x * m for x, m in zip(U, mid)) - 0.5 * (c2 + 0.5 * (K + D) / l) * last
    return torch.stack([first] + mid + [last], -1)


class _Faces:
    """Fluxes through the faces of one direction, in the face frame: what the face
    states give (scalars of each face), then the parts at single velocities."""

    def __init__(self, flux, gas, dt, wL=None, wR=None, half=None):
        self.flux, self.K = flux, gas.K
        if flux == "kfvs":
            self.A, self.B, self.eq = dt, 0.5 * dt * dt, None
            return
        pL, pR = _prims(wL, gas.gamma), _prims(wR, gas.gamma)
        L, _, _, V, xi = _gauss(pL, gas.K)
        w = pL[..., :1] * _mc(L, V, xi, 0, 0, 0)
        _, R, _, V, xi = _gauss(pR, gas.K)
        w = w + pR[..., :1] * _mc(R, V, xi, 0, 0, 0)
        p = self.p = _prims(w, gas.gamma)
        L, R, M, V, xi = _gauss(p, gas.K)
        self.xi2 = xi[2]
        tau = gas.tau(p)
        dts = dt if not torch.is_tensor(dt) else dt[..., 0]
        if flux == "kcu":
            a, b = pL[..., 0] / pL[..., -1], pR[..., 0] / pR[..., -1]
            tau = tau + (a - b).abs() / (a + b) * dts * 2.0
            self.A = tau * (1 - torch.exp(-dts / tau))
            self.m0 = dts - self.A
            self.B = torch.zeros_like(self.A)
            self.eq = (self.m0 * p[..., 0])[..., None] * _mc(M, V, xi, 1, 0, 0)
        else:
            ex = torch.exp(-dts / tau)
            self.A = tau * (1 - ex)
            self.B = -tau * dts * ex + tau * self.A
            self.m0 = dts - self.A
            self.m1 = -tau * self.m0 + self.B
            self.m2 = dts * dts / 2 - tau * self.m0
            self.aL, self.aR = _pdf_slope(p, (w - wL) / half, gas.K), _pdf_slope(p, (wR - w) / half, gas.K)
            t = -p[..., :1] * (_mcs(self.aL, L, V, xi, 1) + _mcs(self.aR, R, V, xi, 1))
            self.aT = _pdf_slope(p, t, gas.K)
            q = lambda x: (x * p[..., 0])[..., None]
            self.eq = q(self.m0) * _mc(M, V, xi, 1, 0, 0) + q(self.m1) * (
                _mcs(self.aL, L, V, xi, 2) + _mcs(self.aR, R, V, xi, 2)) + q(self.m2) * _mcs(self.aT, M, V, xi, 1)
        self.A, self.B = self.A[..., None], self.B[..., None]

    def free(self, up, un, qL, qR, sL, sR):
        return self.A * un * torch.where(up, qL, qR) - self.B * un * un * torch.where(up, sL, sR)

    def equil(self, up, un, ut):
        """fh, fb of the equilibrium part."""
        p = self.p[..., None, :]
        H = _maxwell(p, un, ut)
        B = H * self.K / (2 * p[..., -1])
        if self.flux == "kcu":
            m = self.m0[..., None] * un
            return m * H, m * B
        c2 = un * un if ut is None else un * un + ut * ut
        def poly(a, X, Y):
            a = a[..., None, :]
            s = a[..., 0] + a[..., 1] * un + (a[..., 2] * ut if ut is not None else 0.0)
            return s * X + 0.5 * a[..., -1] * (c2 * X + Y)
        out = []
        for X, Y in ((H, B), (B, self.xi2[..., None] * H)):
            side = torch.where(up, poly(self.aL, X, Y), poly(self.aR, X, Y))
            out.append(self.m0[..., None] * un * X + self.m1[..., None] * un * un * side
                       + self.m2[..., None] * un * poly(self.aT, X, Y))
        return out


def _moments(f, fb, un, ut, wt):
    s = lambda x: (wt * x).sum(-1)
    if ut is None:
        return torch.stack([s(f), s(un * f), 0.5 * (s(un * un * f) + s(fb))], -1)
    return torch.stack([s(f), s(un * f), s(ut * f), 0.5 * (s((un * un + ut * ut) * f) + s(fb))], -1)


def _heat(p, h, b, u, v, wt):
    """Heat flux of each cell: one component, or two."""
    c = [u - p[..., None, 1]] + ([v - p[..., None, 2]] if v is not None else [])
    c2 = sum(x * x for x in c)
    return [0.5 * ((wt * x * c2 * h).sum(-1) + (wt * x * b).sum(-1)) for x in c]


def _shakhov(gas, p, q, u, v):
    pp = p[..., None, :]
    c = [u - pp[..., 1]] + ([v - pp[..., 2]] if v is not None else [])
    c2 = sum(x * x for x in c)
    H = _maxwell(pp, u, v)
    B = H * gas.K / (2 * pp[..., -1])
    f = 0.8 * (1 - gas.Pr) * pp[..., -1] ** 2 / pp[..., 0] * sum(x * y[..., None] for x, y in zip(c, q))
    return f * (2 * pp[..., -1] * c2 + gas.K - 5) * H, f * (2 * pp[..., -1] * c2 + gas.K - 3) * B


def _lines(cfgs, prims, steps, adaptive=False, dev="cuda"):
    """1D solves with held ends, all at once: padded to one size, [solve, cell, velocity]."""
    n, nx, nu = len(cfgs), max(c["nx"] for c in cfgs), max(c["nu"] for c in cfgs)
    P = np.tile(np.array([1.0, 0.0, 1.0]), (n, nx, 1))
    U, W, keep = np.zeros((n, 1, nu)), np.zeros((n, 1, nu)), np.zeros((n, nx, 1), dtype=bool)
    for i, (c, p) in enumerate(zip(cfgs, prims)):
        P[i, :c["nx"]] = p
        U[i, 0, :c["nu"]], W[i, 0, :c["nu"]] = _grid1(c)
        keep[i, 1:c["nx"] - 1] = True
    t = lambda a: torch.from_numpy(a).to(dev)
    p, u, wt, keep = t(P), t(U), t(W), t(keep)
    col = lambda f: torch.tensor([f(c) for c in cfgs], dtype=torch.float64, device=dev)[:, None, None]
    gas = _Gas(cfgs[0], 1)
    gas.mu = col(lambda c: _Gas(c, 1).mu)[..., 0]
    dx, umax = col(lambda c: (c["x1"] - c["x0"]) / c["nx"]), col(lambda c: c["umax"])
    real = torch.arange(nx, device=dev)[None, :] < torch.tensor([c["nx"] for c in cfgs], device=dev)[:, None]
    w = _cons(p, gas.gamma)
    h = _maxwell(p[:, :, None], u)
    b = h * gas.K / (2 * p[:, :, None, 2])
    flux, shak = cfgs[0]["flux"], cfgs[0]["collision"] == "shakhov"
    up = u >= 0

    def step_size():
        rate = torch.maximum(umax[..., 0], p[..., 1].abs()) + torch.sqrt(0.5 * gas.gamma / p[..., 2])
        return 0.5 * dx / torch.where(real, rate, torch.zeros_like(rate)).amax(1)[:, None, None]

    dt = step_size()
    for _ in range(steps):
        if adaptive:
            dt = step_size()
        sh, sb = (_limited(q, dx, False) * keep for q in (h, b))
        half = 0.5 * dx
        if flux == "kfvs":
            F = _Faces(flux, gas, dt)
        else:
            sw = _limited(w, dx, False) * keep
            F = _Faces(flux, gas, dt, (w + half * sw)[:, :-1], (w - half * sw)[:, 1:], half)
        fh = F.free(up, u, (h + half * sh)[:, :-1], (h - half * sh)[:, 1:], sh[:, :-1], sh[:, 1:])
        fb = F.free(up, u, (b + half * sb)[:, :-1], (b - half * sb)[:, 1:], sb[:, :-1], sb[:, 1:])
        fw = _moments(fh, fb, u, None, wt)
        if F.eq is not None:
            fw = fw + F.eq
            eh, eb = F.equil(up, u, None)
            fh, fb = fh + eh, fb + eb
        S = _shakhov(gas, p, _heat(p, h, b, u, None, wt), u, None) if shak else (0.0, 0.0)
        inner = keep[:, 1:-1]
        wn, pn = w.clone(), p.clone()
        wn[:, 1:-1] = w[:, 1:-1] + (fw[:, :-1] - fw[:, 1:]) / dx
        wn = torch.where(keep, wn, w)
        pn = torch.where(keep, _prims(wn, gas.gamma), p)
        r = (dt[..., 0] / gas.tau(pn))[:, 1:-1, None]
        H = _maxwell(pn[:, :, None], u)
        B = H * gas.K / (2 * pn[:, :, None, 2]) + S[1]
        H = H + S[0]
        for q, f, M in ((h, fh, H), (b, fb, B)):
            new = (q[:, 1:-1] + (f[:, :-1] - f[:, 1:]) / dx + r * M[:, 1:-1]) / (1 + r)
            q[:, 1:-1] = torch.where(inner, new, q[:, 1:-1])
        w, p = wn, pn
    return [dict(w=w[i, :c["nx"]], prim=p[i, :c["nx"]], h=h[i, :c["nx"], :c["nu"]], b=b[i, :c["nx"], :c["nu"]])
            for i, c in enumerate(cfgs)]


def _plane(cfg, steps, state, dev="cuda"):
    """A 2D solve; state = (w, prim) or (w, prim, h, b) over all cells incl. ghosts.
    Velocities are taken a block at a time: given the faces' scalars they are independent."""
    gas = _Gas(cfg, 2)
    g, bc, flux, shak = cfg["nxg"], cfg["boundary"], cfg["flux"], cfg["collision"] == "shakhov"
    nx, ny = cfg["nx"], cfg["ny"]
    dx, dy = 1.0 / nx, 1.0 / ny
    u, v, wt = _grid2(cfg, dev)
    shape = (ny + 2 * g, nx + 2 * g)
    w, p = (x.reshape(shape + (4,)).clone() for x in state[:2])
    nv = len(u)
    block = max(1, min(nv, int(4e7 / (shape[0] * shape[1]))))
    parts = [slice(k, min(k + block, nv)) for k in range(0, nv, block)]
    if len(state) == 4:
        h, b = (x.reshape(shape + (nv,)).clone() for x in state[2:])
    else:
        h, b = (torch.empty(shape + (nv,), dtype=torch.float64, device=dev) for _ in range(2))
        for s in parts:
            h[..., s] = _maxwell(p[:, :, None], u[s], v[s])
            b[..., s] = h[..., s] * gas.K / (2 * p[:, :, None, 3])
    inner = p[g:g + ny, g:g + nx]
    sos = torch.sqrt(0.5 * gas.gamma / inner[..., 3])
    rate = (torch.clamp(inner[..., 1].abs(), min=cfg["umax"]) + sos) / dx + (torch.clamp(inner[..., 2].abs(), min=cfg["vmax"]) + sos) / dy
    dt = cfg["cfl"] / float(rate.max())
    # per direction: cells as [line, cell along, ...], face-frame velocities, spacing, face length, n of cells
    view = [lambda q: q[g:g + ny], lambda q: q[:, g:g + nx].transpose(0, 1)]
    vel = [lambda s: (u[s], v[s]), lambda s: (v[s], -u[s])]
    size, length, count = [dx, dy], [dy, dx], [nx, ny]
    turn = [lambda q: q, lambda q: torch.stack([q[..., 0], q[..., 2], -q[..., 1], q[..., 3]], -1)]
    back = [lambda q: q, lambda q: torch.stack([q[..., 0], -q[..., 2], q[..., 1], q[..., 3]], -1)]
    walls = [torch.from_numpy(x).to(dev) for x in _walls(cfg)] if bc == "maxwell" else None
    sw = [torch.zeros(shape + (4,), dtype=torch.float64, device=dev) for _ in range(2)]

    def sided(q, d, n):
        s = torch.zeros_like(q)
        s[:, g:g + n] = _limited(q[:, g:g + n], size[d], True)
        return s

    def pair(x, n):
        return (x[:, g - 1:g + n], x[:, g:g + n + 1]) if g else (x[:, :-1], x[:, 1:])

    def pad(f):
        if g:
            return f
        out = torch.zeros((f.shape[0], f.shape[1] + 2) + f.shape[2:], dtype=f.dtype, device=dev)
        out[:, 1:-1] = f
        return out

    def free(F, d, s):
        un, ut = vel[d](s)
        up, out = un >= 0, []
        for q in (h, b):
            q = view[d](q[..., s])
            sl = sided(q, d, count[d])
            (qL, qR), (sL, sR) = pair(q, count[d]), pair(sl, count[d])
            out.append(F.free(up, un, qL + 0.5 * size[d] * sL, qR - 0.5 * size[d] * sR, sL, sR))
        return un, ut, up, out

    def wall_sum(d, end, rho):
        """Diffuse wall at one end of direction d: its density, or with it fw."""
        bcp = turn[d](walls[2 * d + end])
        total = [0.0, 0.0] if rho is None else torch.zeros((bcp.shape[0], 4), dtype=torch.float64, device=dev)
        for s in parts:
            un, ut = vel[d](s)
            into = un >= 0 if end == 0 else -un >= 0
            q = view[d](h[..., s])[:, 0 if end == 0 else -1]
            unit = bcp.clone()
            unit[:, 0] = 1.0 if rho is None else rho
            H = _maxwell(unit[:, None], un, ut)
            if rho is None:
                total[0] = total[0] + (wt[s] * un * q * ~into).sum(-1)
                total[1] = total[1] + (wt[s] * un * H * into).sum(-1)
                continue
            qb = view[d](b[..., s])[:, 0 if end == 0 else -1]
            fh = un * torch.where(into, H, q)
            fb = un * torch.where(into, H * gas.K / (2 * unit[:, None, 3]), qb)
            total += _moments(fh, fb, un, ut, wt[s])
        return -total[0] / total[1] if rho is None else total * dt * length[d]

    for _ in range(steps):
        F, fw, rhos = [], [], {}
        for d in range(2):
            sw[d] = sw[d].clone()
            view[d](sw[d])[:, g:g + count[d]] = _limited(view[d](w)[:, g:g + count[d]], size[d], True)
            if flux == "kfvs":
                F.append(_Faces(flux, gas, dt))
            else:
                (wl, wr), (sl, sr) = pair(view[d](w), count[d]), pair(view[d](sw[d]), count[d])
                half = 0.5 * size[d]
                F.append(_Faces(flux, gas, dt, turn[d](wl + half * sl), turn[d](wr - half * sr), half))
            total = 0.0 if F[d].eq is None else F[d].eq
            for s in parts:
                un, ut, _, (fh, fb) = free(F[d], d, s)
                total = total + _moments(fh, fb, un, ut, wt[s])
            total = pad(total * length[d])
            if walls is not None:
                for end in (0, 1):
                    rhos[d, end] = wall_sum(d, end, None)
                    total[:, 0 if end == 0 else -1] = wall_sum(d, end, rhos[d, end])
            fw.append(back[d](total))
        if shak:
            q = [0.0, 0.0]
            for s in parts:
                q = [x + y for x, y in zip(q, _heat(p, h[..., s], b[..., s], u[s], v[s], wt[s]))]
        old = p
        diff = fw[0][:, :-1] - fw[0][:, 1:] + (fw[1][:, :-1] - fw[1][:, 1:]).transpose(0, 1)
        w = w.clone()
        at = slice(1, -1) if bc == "fix" else slice(None)  # held boundary cells
        cells = (slice(g, g + ny), slice(g, g + nx))
        w[cells][at, at] += diff[at, at] / (dx * dy)
        p = p.clone()
        p[cells][at, at] = _prims(w[cells][at, at], gas.gamma)
        r = (dt / gas.tau(p[cells][at, at]))[..., None]
        for s in parts:
            df = [0.0, 0.0]
            for d in range(2):
                un, ut, up, f = free(F[d], d, s)
                if flux != "kfvs":
                    f = [x + y for x, y in zip(f, F[d].equil(up, un, ut))]
                for k in range(2):
                    t = pad(f[k] * length[d])
                    if walls is not None:
                        for end in (0, 1):
                            e = 0 if end == 0 else -1
                            into = un >= 0 if end == 0 else -un >= 0
                            m = turn[d](walls[2 * d + end]).clone()
                            m[:, 0] = rhos[d, end]
                            M = _maxwell(m[:, None], un, ut)
                            M = M if k == 0 else M * gas.K / (2 * m[:, None, 3])
                            t[:, e] = un * torch.where(into, M, view[d]((h, b)[k][..., s])[:, e]) * length[d] * dt
                    t = t[:, :-1] - t[:, 1:]
                    df[k] = df[k] + (t if d == 0 else t.transpose(0, 1))
            pn = p[cells][at, at]
            H = _maxwell(pn[:, :, None], u[s], v[s])
            M = [H, H * gas.K / (2 * pn[:, :, None, 3])]
            if shak:
                S = _shakhov(gas, old[cells][at, at], [x[cells][at, at] for x in q], u[s], v[s])
                M = [x + y for x, y in zip(M, S)]
            for k, q_ in enumerate((h, b)):
                c = q_[cells][at, at][..., s]
                q_[cells][at, at][..., s] = (c + df[k][at, at] / (dx * dy) + r * M[k]) / (1 + r)
        if bc == "extra":
            for q_ in (w, p, h, b, sw[0], sw[1]):
                q_[:, 0], q_[:, -1] = q_[:, 1], q_[:, -2]
                q_[0], q_[-1] = q_[1], q_[-2]
    flat = lambda x: x.reshape(-1, x.shape[-1])
    return dict(w=flat(w), prim=flat(p), h=flat(h), b=flat(b))


def _edges(points, cells):
    """Faces of a triangle mesh in plain numpy: pairs of cells, normals from the first
    to the second of length |d| / (|d| + 1e-6), lengths; faces, orientations and
    neighbours of each cell; areas; smallest centre-to-edge distances."""
    n = len(cells)
    a, b = cells.reshape(-1), cells[:, [1, 2, 0]].reshape(-1)
    key = np.minimum(a, b).astype(np.int64) * (len(points) + 1) + np.maximum(a, b)
    _, first, inv = np.unique(key, return_index=True, return_inverse=True)
    inv = inv.reshape(-1)
    owner = np.arange(3 * n) // 3
    c1, c2 = first // 3, np.full(len(first), -1)
    later = np.arange(3 * n) != first[inv]
    c2[inv[later]] = owner[later]
    center = points[cells].mean(1)
    pa, pb = points[a[first]], points[b[first]]
    d = pb - pa
    ln = np.sqrt((d * d).sum(1))
    nrm = np.stack([-d[:, 1], d[:, 0]], 1) / (ln + 1e-6)[:, None]
    to = np.where((c2 >= 0)[:, None], center[c2] - center[c1], center[c1] - 0.5 * (pa + pb))
    nrm[(nrm * to).sum(1) < 0] *= -1
    cf = inv.reshape(n, 3)
    sign = np.where(c1[cf] == np.arange(n)[:, None], 1.0, -1.0)
    nb = np.where(sign > 0, c2[cf], c1[cf])
    p, q, r = (points[cells[:, k]] for k in range(3))
    area = 0.5 * np.abs((q[:, 0] - p[:, 0]) * (r[:, 1] - p[:, 1]) - (r[:, 0] - p[:, 0]) * (q[:, 1] - p[:, 1]))
    A, B, C = points[a].reshape(n, 3, 2), points[b].reshape(n, 3, 2), center[:, None]
    dist = np.abs((B[..., 0] - A[..., 0]) * (A[..., 1] - C[..., 1]) - (A[..., 0] - C[..., 0]) * (B[..., 1] - A[..., 1]))
    dist = dist / np.sqrt(((B - A) ** 2).sum(-1) + 1e-6)
    return c1, c2, nrm, ln, cf, sign, nb, area, dist.min(1), center


def _triangles(case, seed, dev="cuda"):
    points, cells = _mesh_points(case)
    c1, c2, nrm, ln, cf, sign, nb, area, dmin, center = _edges(points, cells)
    w, p, h, b = _mesh_state(center, case, seed, dev)
    gas = _Gas(dict(inK=1.0, prandtl=2.0 / 3.0, omega=0.72, alphaRef=1.0, omegaRef=0.5, knudsen=0.075), 2)
    u, v, wt = _grid2(dict(umin=-5.0, umax=5.0, nu=case["nu"], vmin=-5.0, vmax=5.0, nv=case["nv"], vMeshType="rectangle"), dev)
    missing = (nb < 0).sum(1)
    mean, free = np.nonzero(missing == 1)[0], missing == 0  # boundary cells: mean of two, corners held
    level = {}
    for c in mean:  # a later one of these sees an earlier one's new value
        level[c] = 1 + max([level[x] for x in nb[c] if x >= 0 and x < c and x in level] + [0])
    order = [np.array([c for c in mean if level[c] == k]) for k in range(1, max(level.values(), default=0) + 1)]
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)
    pairs = [np.array([[x for x in nb[c] if x >= 0] for c in cs]) for cs in order]
    order, pairs = [t(x) for x in order], [t(x) for x in pairs]
    inside = t((c2 >= 0).astype(np.float64))[:, None]
    i1, i2 = t(c1), t(np.maximum(c2, 0))
    n1, n2, ln, cf, sign, area, free = t(nrm[:, :1]), t(nrm[:, 1:]), t(ln[:, None]), t(cf), t(sign), t(area[:, None]), t(free)[:, None]
    um = 5.0 + torch.sqrt(0.5 * gas.gamma / p[:, 3])
    dt = 0.5 / float((torch.sqrt(um * um + um * um) / t(dmin)).max())
    un, ut = u * n1 + v * n2, v * n1 - u * n2
    up = un >= 0
    across = lambda f: sum(f[cf[:, k]] * sign[:, k:k + 1] for k in range(3)) / area
    for _ in range(case["steps"]):
        fh, fb = (dt * un * torch.where(up, q[i1], q[i2]) * ln * inside for q in (h, b))
        m = _moments(fh, fb, un, ut, wt)
        fw = torch.cat([m[:, :1], m[:, 1:2] * n1 - m[:, 2:3] * n2, m[:, 1:2] * n2 + m[:, 2:3] * n1, m[:, 3:]], 1)
        S = _shakhov(gas, p, _heat(p, h, b, u, v, wt), u, v) if case["coll"] == "shakhov" else (0.0, 0.0)
        w = torch.where(free, w - across(fw), w)
        p = torch.where(free, _prims(w, gas.gamma), p)
        r = (dt / gas.tau(p))[:, None]
        H = _maxwell(p[:, None], u, v)
        B = H * gas.K / (2 * p[:, 3:]) + S[1]
        H = H + S[0]
        h, b = (torch.where(free, (q - across(f) + r * M) / (1 + r), q) for q, f, M in ((h, fh, H), (b, fb, B)))
        for cs, ps in zip(order, pairs):
            for q in (w, h, b):
                q[cs] = 0.5 * (q[ps[:, 0]] + q[ps[:, 1]])
            p[cs] = _prims(w[cs], gas.gamma)
    return dict(w=w, prim=p, h=h, b=b)


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    k, n = case["kind"], case["steps"]
    if k in ("adaptive", "line"):
        cfg = _cfg_line(case)
        return _lines([cfg], [_line_prim(cfg, seed)], n, k == "adaptive")[0]
    if k in ("plane", "restart"):
        cfg = _cfg_plane(case)
        if k == "restart":
            return _plane(cfg, n, _restart_state(cfg, case, seed, "cuda"))
        p = torch.from_numpy(_plane_prim(cfg, seed)).cuda()
        out = _plane(cfg, n, (_cons(p, _gamma(cfg["inK"], 2)), p))
        return out if case["full"] else {q: out[q] for q in ("w", "prim")}
    if k == "shocks":
        cfgs = _cfg_shocks(case, seed)
        out = _lines(cfgs, _shock_prims(cfgs), n)
        return {q: torch.cat([x[q] for x in out]) for q in ("w", "prim")}
    if k == "mesh":
        out = _triangles(case, seed)
        return out if case["full"] else {q: out[q] for q in ("w", "prim")}
    lines, planes = _cfg_serve(case, seed)
    out = []
    for c in lines:
        x = np.arange(c["nx"]) + 0.5 <= 0.5 * c["nx"]
        out += _lines([c], [np.where(x[:, None], [1.0, 0.0, 0.5], [0.125, 0.0, 0.625])], n)
    for c in planes:
        p = torch.tensor([1.0, 0.0, 0.0, 1.0], dtype=torch.float64, device="cuda").expand(c["ny"], c["nx"], 4)
        out.append(_plane(c, n, (_cons(p, _gamma(1.0, 2)), p)))
    return {q: [x[q] for x in out] for q in ("prim", "w")}
