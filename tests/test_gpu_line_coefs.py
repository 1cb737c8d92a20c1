"""The relaxation factors of a single FP32 line's cells (kb_batch.cuh): FP64 until
one rounding, as the general form's."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "kb_batch.cuh"
using namespace kb;
__global__ void k(int n, const double* a, const double* b, const double* c, const double* d, float* o, float om1) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  seg_relax(a[i], b[i], (float)c[i], om1, o[3 * i], o[3 * i + 1]);
  o[3 * i + 2] = seg_heat(a[i], b[i], c[i], d[i]);
}
extern "C" int go(int n, const double* in, float* out, float om1) {
  double* d;
  if (cudaMalloc(&d, 44L * n) != cudaSuccess) return 1;
  cudaMemcpy(d, in, 32L * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(n, d, d + n, d + 2L * n, d + 3L * n, (float*)(d + 4L * n), om1);
  cudaMemcpy(out, d + 4L * n, 12L * n, cudaMemcpyDeviceToHost);
  int rc = (int)cudaGetLastError();
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    from kitgpu import build
    d = tmp_path_factory.mktemp("coefs")
    src, so = str(d / "c.cu"), str(d / "c.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                                                  build.INCLUDE, "-shared", "-Xcompiler", "-fPIC", "-o", so, src], check=True)
    return ctypes.CDLL(so)


def _call(lib, a, b, c, d, om1):
    x, o = np.concatenate([a, b, c, d]), np.zeros((len(a), 3), np.float32)
    assert lib.go(len(a), x.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), o.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                  ctypes.c_float(om1)) == 0
    return o


def test_one_rounding_to_fp32(lib):
    """omega = 1: no power, so each factor is within half a unit of the exact one,
    1 / (1 + dt / tau) of the rounded dt / tau (and of the few FP64 roundings
    before it, 2^-49)."""
    rng = np.random.default_rng(1)
    a, b, c, d = (10.0 ** rng.uniform(-e, e, 20000) for e in (6, 2, 2, 3))
    o = _call(lib, a, b, c, d, 0.0)
    for got, want in ((o[:, 0], a * b), (o[:, 1], 1.0 / (1.0 + o[:, 0].astype(np.float64))), (o[:, 2], a * (b * b) / c * d)):
        half = 0.5 * np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
        assert np.all(np.abs(got.astype(np.float64) - want) <= half * (1 + 1e-6) + 2.0 ** -49 * want)


def test_power_of_the_collision_time(lib):
    """dt / tau with its power in FP32: two units more for powf, and the rounding
    of lambda (half a unit times 1 - omega)."""
    rng = np.random.default_rng(2)
    a, b, c, d = (10.0 ** rng.uniform(-e, e, 20000) for e in (6, 2, 2, 3))
    for om in (0.5, 0.72, 0.81):
        o = _call(lib, a, b, c, d, om - 1.0)
        want = a * b * c ** float(np.float32(om - 1.0))
        assert np.max(np.abs(o[:, 0] / want - 1.0)) < (0.5 + 2.0 + 0.5) * 2.0 ** -23
