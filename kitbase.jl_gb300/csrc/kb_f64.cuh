// kb_f64.cuh -- FP64 arithmetic of the hot loops.  GB300 issues FP64 at 1/64
// of its FP32 rate (two lanes per clock and multiprocessor), so the FP64 forms
// are bound by the number of FP64 instructions: a division costs about ten.
#pragma once

#include <cuda_runtime.h>

namespace kb {

// 1 / x to about one unit in the last place for positive normal x: the PTX
// approximation (rcp.approx.ftz.f64, about 20 bits) and one third-order Newton
// (Halley) step, r (1 + e + e^2) with e = 1 - x r, whose error is e^3.
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// van Leer slope times dx from raw differences: (a|b| + b|a|) / (|a| + |b| + eps)
// (src/Reconstruction/recon_limiter.jl:17-19).  The denominator is at least
// eps = 1e-7 dx > 0.
__device__ __forceinline__ double vl64(double qm, double q0, double qp, double eps) {
  const double a = q0 - qm, b = qp - q0;
  const double d = (fabs(a) + fabs(b)) + eps;
  return fma(a, fabs(b), b * fabs(a)) * rcp64(d);
}

}  // namespace kb
