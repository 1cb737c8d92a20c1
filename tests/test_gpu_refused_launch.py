"""A step whose kernel launch the runtime refuses: the call returns an error and
the handle keeps the state it had.  The refusal is made on the host, in a child
process: a preloaded cudaLaunchKernelExC gives the runtime one launch of more
threads per block than any device takes, which it answers with an error code."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#include <cuda_runtime_api.h>
static int countdown = -1;
void refuse_after(int n) { countdown = n; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  static cudaError_t (*next)(const cudaLaunchConfig_t*, const void*, void**);
  if (!next) {  // (loaded with the library, outside the global search order)
    char name[32];
    snprintf(name, sizeof name, "libcudart.so.%d", CUDART_VERSION / 1000);
    void* rt = dlopen(name, RTLD_LAZY | RTLD_NOLOAD);
    if (!rt || !(*(void**)&next = dlsym(rt, "cudaLaunchKernelExC"))) abort();
  }
  if (countdown >= 0 && countdown-- == 0) {
    cudaLaunchConfig_t d = *c;
    d.blockDim.x = 1 << 20;
    return next(&d, f, a);
  }
  return next(c, f, a);
}
"""

CHILD = r"""
import ctypes, os, sys
import numpy as np
import kitgpu
from kitgpu import batch as KB, unstruct as US
from kitgpu._native import KitGPUError
from cases import sod, shock
shim = ctypes.CDLL(os.environ["LD_PRELOAD"])
kind, prec, nsteps = sys.argv[1], sys.argv[2], int(sys.argv[3])

def make():
    if kind == "line":
        KS, ctr, f, t = kitgpu.initialize(sod(nx=20, nu=17), precision=prec)
        return ctr.handle, 1e-3
    if kind == "mesh":
        from test_gpu_unstruct import _setup
        hd = US.init_fvm(_setup(dict(boundary="extra", collision="bgk", nx=5, ny=4, nu=6, nv=6, jitter=0.2))[0], prec)
        return hd, 1e-3
    b = KB.Batch(KB.solver_sets([KB.shock_config(2.0, 20, 18), KB.shock_config(3.0, 31, 24)]), prec)
    b.init_initial()
    b.timestep()
    return b, None

def step(h, dt, n):
    return h.step(n) if dt is None else h.step(dt, n)

def state(h):
    s = h.download()
    return [x[k] for x in (s if isinstance(s, list) else [s]) for k in ("w", "prim", "h", "b")]

a, dt = make()
step(a, dt, 3)
before = state(a)
shim.refuse_after(0)
try:
    step(a, dt, nsteps)
    sys.exit("no error from a refused launch")
except KitGPUError as e:
    assert e.code == -3, e
shim.refuse_after(-1)
assert all(np.array_equal(x, y) for x, y in zip(state(a), before)), "the state changed"
step(a, dt, nsteps)
b, dt = make()
step(b, dt, 3)
step(b, dt, nsteps)
assert all(np.array_equal(x, y) for x, y in zip(state(a), state(b))), "later steps differ"
print("ok")
"""


@pytest.fixture(scope="module")
def shim(gpu_lib, tmp_path_factory):
    from kitgpu import build
    d = tmp_path_factory.mktemp("shim")
    src, so = str(d / "shim.c"), str(d / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O2", "-I", inc, "-o", so, src, "-ldl"], check=True)
    return so


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,nsteps", [("line", 1), ("mesh", 1), ("batch", 1), ("batch", 8)])
def test_refused_launch_is_an_error(shim, kind, nsteps, prec):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = [os.path.join(root, p) for p in ("tests", "kitbase.jl_gb300", "oracle")]
    env = dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=os.pathsep.join(path))
    r = subprocess.run([sys.executable, "-c", CHILD, kind, prec, str(nsteps)], env=env, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
