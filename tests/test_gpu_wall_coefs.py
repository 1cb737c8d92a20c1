"""The FP32 form's wall Maxwellian (kb_wall.cuh): its exponent is formed in FP64
and rounded once."""
import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include "kb_wall.cuh"
using namespace kb;
__global__ void k(int n, const double* a, float* o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 E = maxwell_exp2(a[i], a[n + i], a[2 * n + i], a[3 * n + i], EXP64_TAB);
  o[4 * i] = E.x;
  o[4 * i + 1] = E.y;
  o[4 * i + 2] = E.z;
  o[4 * i + 3] = E.w;
}
extern "C" int go(int n, const double* in, float* out) {
  double* d;
  if (cudaMalloc(&d, 48L * n) != cudaSuccess) return 1;
  cudaMemcpy(d, in, 32L * n, cudaMemcpyHostToDevice);
  k<<<(n + 127) / 128, 128>>>(n, d, (float*)(d + 4L * n));
  cudaMemcpy(out, d + 4L * n, 16L * n, cudaMemcpyDeviceToHost);
  int rc = (int)cudaGetLastError();
  cudaFree(d);
  return rc;
}
"""


def test_wall_exponent_rounds_once(gpu_lib, tmp_path):
    """Densities over 14 decades: each term within half a unit of the exact one,
    and 2^-50 of its parts (the FP64 roundings before)."""
    from kitgpu import build
    src, so = str(tmp_path / "w.cu"), str(tmp_path / "w.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                                                  build.INCLUDE, "-shared", "-Xcompiler", "-fPIC", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)
    n = 20000
    rng = np.random.default_rng(1)
    r = 10.0 ** rng.uniform(-7, 7, n)
    r[:3] = [1.0, 1.0 + 2.0 ** -30, 2.0]
    U, V = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    lam = 10.0 ** rng.uniform(-1, 1, n)
    U[:3] = V[:3] = 0.0
    x, o = np.concatenate([r, U, V, lam]), np.zeros((n, 4), np.float32)
    assert lib.go(n, x.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), o.ctypes.data_as(ctypes.POINTER(ctypes.c_float))) == 0
    L = 1.442695040888963407359924681001892137
    ll = np.longdouble(lam) * L
    a, b = np.log2(np.longdouble(r)), ll * (np.longdouble(U) ** 2 + np.longdouble(V) ** 2)
    for k, (want, parts) in enumerate([(a - b, abs(a) + b + 1.0), (2 * ll * U, 0), (2 * ll * V, 0), (-ll, 0)]):
        half = 0.5 * np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
        assert np.all(np.abs(o[:, k] - want) <= half * (1 + 1e-6) + 2.0 ** -50 * (parts + np.abs(want))), k
