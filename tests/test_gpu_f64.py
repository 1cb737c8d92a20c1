"""The FP64 forms of kb_f64.cuh (reciprocal, square root, exponentials, power)
against exactly rounded values: each within a few units in the last place."""
import ctypes
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "kb_f64.cuh"
using namespace kb;
__global__ void k(int op, int n, const double* x, const double* y, double* o, Pow64 p) {
  __shared__ double tab[EXP64_N];
  exp64_load(tab, threadIdx.x, blockDim.x);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = op == 0 ? rcp64(x[i]) : op == 1 ? sqrt64(x[i]) : op == 2 ? exp2_tab(x[i], y[i], tab)
       : op == 3 ? pow_tab(x[i], p, tab) : op == 4 ? (double)f32_of(x[i]) : op == 5 ? f64_of((float)x[i])
       : op == 6 ? (pos64(x[i]) ? 1.0 : 0.0) : (nonneg64(x[i]) ? 1.0 : 0.0);
}
extern "C" int go(int op, int n, const double* x, const double* y, double* o, double pw) {
  double *d;
  if (cudaMalloc(&d, 24L * n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, 8L * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, 8L * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(op, n, d, d + n, d + 2L * n, pow64_of(pw));
  cudaMemcpy(o, d + 2L * n, 8L * n, cudaMemcpyDeviceToHost);
  int rc = (int)cudaGetLastError();
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    from kitgpu import build
    d = tmp_path_factory.mktemp("f64")
    src, so = str(d / "f64.cu"), str(d / "f64.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-I", build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                                                  "-o", so, src], check=True)
    return ctypes.CDLL(so)


def ulps(got, exact):
    return max(float(abs(Decimal(g) - e) / Decimal(np.spacing(float(e)).item())) for g, e in zip(got.tolist(), exact))


def call(lib, op, x, y=None, pw=0.0):
    o, D = np.zeros(len(x)), ctypes.POINTER(ctypes.c_double)
    y = np.ones(len(x)) if y is None else y
    assert lib.go(op, len(x), *[a.ctypes.data_as(D) for a in (x, y, o)], ctypes.c_double(pw)) == 0
    return o


# largest error in units in the last place: half a unit for the last rounding
# and about one for each operation before it that acts on the whole value
@pytest.mark.parametrize("name,op,most", [("rcp64", 0, 1.5), ("sqrt64", 1, 2.0)])
def test_division_and_root(lib, name, op, most):
    getcontext().prec = 50
    x = 10.0 ** np.random.default_rng(op).uniform(-200, 200, 2000)
    x[:8] = [1.0, 2.0, 0.5, 1.0 + 2 ** -52, 1.0 - 2 ** -53, 3.0, 0.25, np.sqrt(2.0)]
    X = [Decimal(v) for v in x.tolist()]
    assert ulps(call(lib, op, x), [1 / v for v in X] if op == 0 else [v.sqrt() for v in X]) <= most, name


def test_exp2_tab(lib):
    """2^(x y / 256), x y <= 0, down to the smallest normal result; beyond, 0."""
    getcontext().prec = 50
    rng = np.random.default_rng(2)
    x, y = -10.0 ** rng.uniform(-9, 2.5, 2000), 10.0 ** rng.uniform(-6, 2.8, 2000)
    y[:4], x[4] = 0.0, 0.0
    o = call(lib, 2, x, y)
    e = [Decimal(a) * Decimal(b) / 256 for a, b in zip(x.tolist(), y.tolist())]
    live = [k for k in range(2000) if e[k] > -1020]
    assert ulps(o[live], [(Decimal(2).ln() * e[k]).exp() for k in live]) <= 2.5
    assert all(o[k] == 0.0 for k in range(2000) if e[k] < -1022)


@pytest.mark.parametrize("y", [-0.19, -0.28, -0.5, 0.0, 1.0, -1.0, 0.7, 2.0])
def test_pow_tab(lib, y):
    getcontext().prec = 50
    x = 10.0 ** np.random.default_rng(3).uniform(-30, 30, 1000)
    x[:500] = 10.0 ** np.random.default_rng(4).uniform(-2, 2, 500)
    x[:6] = [1.0, 2.0, 0.5, 1.0 + 2 ** -52, 1.0 - 2 ** -53, np.sqrt(2.0)]
    o = call(lib, 3, x, pw=y)
    X = [Decimal(v) for v in x.tolist()]
    # y j / 256 is rounded in the reduction of large |log x|: 70 / 2^53 more
    assert ulps(o[:500], [(Decimal(y) * v.ln()).exp() for v in X[:500]]) <= 4.0
    assert ulps(o, [(Decimal(y) * v.ln()).exp() for v in X]) <= 4.0 + 70 * abs(y)


def test_integer_forms(lib):
    """Conversions as the hardware rounds them, tests of sign and range."""
    rng = np.random.default_rng(5)
    x = np.concatenate([rng.uniform(-1, 1, 4000) * 10.0 ** rng.integers(-37, 38, 4000),
                        [0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, 1.0 + 2 ** -24, 1.0 + 3 * 2 ** -24, 2.0 ** -126,
                         float(np.finfo(np.float32).max), 3.5e38, -1e300, 1e-300]])
    with np.errstate(over="ignore", under="ignore"):
        f = x.astype(np.float32)
    want = np.where(np.abs(f) < np.finfo(np.float32).tiny, np.copysign(np.float32(0), f), f).astype(np.float64)
    assert np.array_equal(call(lib, 4, x), want)
    assert np.array_equal(call(lib, 5, want), want)
    assert np.isnan(call(lib, 4, np.array([np.nan]))).all() and np.isnan(call(lib, 5, np.array([np.nan]))).all()
    z = np.array([1.0, -1.0, 0.0, -0.0, np.inf, -np.inf, np.nan, 1e-300, 1e300, -1e-300])
    assert call(lib, 6, z).tolist() == [1, 0, 0, 0, 0, 0, 0, 1, 1, 0]
    assert call(lib, 7, z[[0, 1, 2, 7, 9]]).tolist() == [1, 0, 1, 1, 0]
