// kb_f64.cuh -- FP64 arithmetic of the hot loops and of the serial per-cell
// and per-face algebra.
//
// GB300 issues FP64 at 1/64 of its FP32 rate: measured, an FP64 instruction of
// a warp holds its quarter of the multiprocessor for 64 to 76 cycles, whatever
// the number of active lanes, and so does a comparison of doubles and a
// conversion between double and float or int.  All forms here are made for
// few FP64 instructions; tests, conversions and powers of two go through the
// integer pipe.  Measured cycles of one warp: a / b 582, sqrt 600, exp 1115,
// pow 6170 against rcp64 205, sqrt64 345, exp2_tab 550, pow_tab 1250.
// Each is good to a few units in the last place (tests/test_gpu_f64.py).
#pragma once

#include <cuda_runtime.h>

namespace kb {

// ------------------------------------------------------ through the integer pipe

// x > 0, normal and finite
__device__ __forceinline__ bool pos64(double x) {
  return (unsigned)(__double2hiint(x) - 0x00100000) < 0x7fe00000u;
}
// x >= 0 for an x that is not -0 with a meaning of its own: the sign bit
__device__ __forceinline__ bool nonneg64(double x) { return __double2hiint(x) >= 0; }
// (float)x, rounded to nearest even; results below 2^-126 are 0
__device__ __forceinline__ float f32_of(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long a = b & 0x7fffffffffffffffull;
  const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
  unsigned r = (unsigned)((a - (896ull << 52) + 0x0fffffffull + ((a >> 29) & 1ull)) >> 29);
  if (a < (897ull << 52)) r = 0u;
  if (a >= (1151ull << 52)) r = a > (2047ull << 52) ? 0x7fffffffu : 0x7f800000u;
  return __uint_as_float(r | sign);
}
// (double)x; subnormal x are 0
__device__ __forceinline__ double f64_of(float x) {
  const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu;
  unsigned hi = (a >> 3) + (896u << 20);
  if (a >= 0x7f800000u) hi |= 0x7ff00000u;
  if (a < 0x00800000u) return __hiloint2double((int)(b & 0x80000000u), 0);
  return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)(b << 29));
}
// 2^n p for a normal p whose result is normal: added to the exponent field
__device__ __forceinline__ double scale64(double p, int n) {
  return __hiloint2double(__double2hiint(p) + (n << 20), __double2loint(p));
}

// ----------------------------------------------------------- division and roots

// 1 / x of a normal x: the PTX approximation (rcp.approx.ftz.f64, about 20
// bits) and one third-order Newton (Halley) step, r (1 + e + e^2) with
// e = 1 - x r, whose error is e^3.
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// sqrt(x) of a positive normal x: x r with r ~ 1 / sqrt(x) (rsqrt.approx.ftz.f64,
// about 20 bits) and the third-order step y (1 + e / 2 + 3 e^2 / 8),
// e = 1 - x r^2.
__device__ __forceinline__ double sqrt64(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double y = x * r;
  const double e = fma(-y, r, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// van Leer slope times dx from raw differences: (a|b| + b|a|) / (|a| + |b| + eps)
// (src/Reconstruction/recon_limiter.jl:17-19).  The denominator is at least
// eps = 1e-7 dx > 0.
__device__ __forceinline__ double vl64(double qm, double q0, double qp, double eps) {
  const double a = q0 - qm, b = qp - q0;
  const double d = (fabs(a) + fabs(b)) + eps;
  return fma(a, fabs(b), b * fabs(a)) * rcp64(d);
}

// -------------------------------------------------------- exponentials, powers

// Powers of two by a table of 2^(j / 256) (a copy in shared memory) and a
// polynomial of degree 4 in the remaining fraction f, |f| <= 1/2 of a 256th
// (Tang's table-driven form; the remainder is 4e-17).
constexpr int EXP64_N = 256;
// (ln 2 / 256)^i / i!
constexpr double EXP64_K1 = 0x1.62e42fefa39efp-9, EXP64_K2 = 0x1.ebfbdff82c58fp-19,
                 EXP64_K3 = 0x1.c6b08d704a0c0p-29, EXP64_K4 = 0x1.3b2ab6fba4e77p-39;
static __device__ const double EXP64_TAB[EXP64_N] = {
    0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0, 0x1.02168143b0281p+0,
    0x1.02c9a3e778061p+0, 0x1.037d42e11bbccp+0, 0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0,
    0x1.059b0d3158574p+0, 0x1.0650a0e3c1f89p+0, 0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0,
    0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0, 0x1.0a9c79b1f3919p+0,
    0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0, 0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0,
    0x1.0e3ec32d3d1a2p+0, 0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0,
    0x1.11301d0125b51p+0, 0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0, 0x1.136a814f204abp+0,
    0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0, 0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0,
    0x1.172b83c7d517bp+0, 0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0, 0x1.1972658375d2fp+0,
    0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0, 0x1.1c82f95281c6bp+0,
    0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0, 0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0,
    0x1.2063b88628cd6p+0, 0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0,
    0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0, 0x1.251ce4fb2a63fp+0, 0x1.25e85711ece75p+0,
    0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0, 0x1.284dfe1f56381p+0, 0x1.291ba7591bb70p+0,
    0x1.29e9df51fdee1p+0, 0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
    0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0, 0x1.2f9d24abd886bp+0,
    0x1.306fe0a31b715p+0, 0x1.31432edeeb2fdp+0, 0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0,
    0x1.33c08b26416ffp+0, 0x1.3496266e3fa2dp+0, 0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0,
    0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0, 0x1.39a401b7140efp+0,
    0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0, 0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0,
    0x1.3dea64c123422p+0, 0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0,
    0x1.4160a21f72e2ap+0, 0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0, 0x1.43ffa3f84b9d4p+0,
    0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0, 0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0,
    0x1.486a2b5c13cd0p+0, 0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0, 0x1.4b17dea6db7d7p+0,
    0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0, 0x1.4eb2d81d8abffp+0,
    0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0, 0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0,
    0x1.5342b569d4f82p+0, 0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0,
    0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0, 0x1.58d12d497c7fdp+0, 0x1.59c0827ff07ccp+0,
    0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0, 0x1.5c9268a5946b7p+0, 0x1.5d84590998b93p+0,
    0x1.5e76f15ad2148p+0, 0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
    0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0, 0x1.652b9febc8fb7p+0,
    0x1.6623882552225p+0, 0x1.671c1c70833f6p+0, 0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6b052fa75173ep+0, 0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0,
    0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0, 0x1.70f7466f42e87p+0,
    0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0, 0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0,
    0x1.75feb564267c9p+0, 0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0,
    0x1.7a11473eb0187p+0, 0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0, 0x1.7d26a62ff86f0p+0,
    0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0, 0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0,
    0x1.82589994cce13p+0, 0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0, 0x1.857f4179f5b21p+0,
    0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0, 0x1.89bd0a478580fp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0, 0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0,
    0x1.8f1ae99157736p+0, 0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0,
    0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0, 0x1.95a44cbc8520fp+0, 0x1.96bdd9a7670b3p+0,
    0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0, 0x1.9a0f170ca07bap+0, 0x1.9b2bb4d53fe0dp+0,
    0x1.9c49182a3f090p+0, 0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
    0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0, 0x1.a42c980460ad8p+0,
    0x1.a5503b23e255dp+0, 0x1.a674a8af46052p+0, 0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0,
    0x1.a9e6b5579fdbfp+0, 0x1.ab0e521356ebap+0, 0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0,
    0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0, 0x1.b20ce6c9a8952p+0,
    0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0, 0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0,
    0x1.b7f76f2fb5e47p+0, 0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0,
    0x1.bcc1e904bc1d2p+0, 0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0, 0x1.c06286141b33dp+0,
    0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0, 0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0,
    0x1.c67f12e57d14bp+0, 0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0, 0x1.ca3405751c4dbp+0,
    0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0, 0x1.cf3155b5bab74p+0,
    0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0, 0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0,
    0x1.d5818dcfba487p+0, 0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0,
    0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0, 0x1.dd321f301b460p+0, 0x1.de7d5641c0658p+0,
    0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0, 0x1.e264614f5a129p+0, 0x1.e3b333b16ee12p+0,
    0x1.e502ee78b3ff6p+0, 0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
    0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0, 0x1.ee4aaa2188510p+0,
    0x1.efa1bee615a27p+0, 0x1.f0f9c1cb6412ap+0, 0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0,
    0x1.f50765b6e4540p+0, 0x1.f6632798844f8p+0, 0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0,
    0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0, 0x1.fe9d96b2a23d9p+0};
__device__ __forceinline__ void exp64_load(double* tab, int tid, int nthreads) {
  for (int j = tid; j < EXP64_N; j += nthreads) tab[j] = EXP64_TAB[j];
}
// Splits a b into an integer n (nearest) and the fraction f, both exact: adding
// 1.5 2^52 leaves n in the low word.
__device__ __forceinline__ int split64(double a, double b, double& f) {
  constexpr double big = 6755399441055744.0;
  const double t = fma(a, b, big);
  f = fma(a, b, -(t - big));
  return __double2loint(t);
}
// 2^(f / 256) - 1
__device__ __forceinline__ double exp64_poly(double f) {
  return f * fma(fma(fma(EXP64_K4, f, EXP64_K3), f, EXP64_K2), f, EXP64_K1);
}
// 2^(a b / 256): 8 FP64 instructions.  Results below 2^-1021 are 0, those from
// 2^1023 up infinite, and not a number stays so.  The range is judged on the
// whole pattern of t = a b + 1.5 2^52, which grows with t from one infinity to
// the other (on each side of zero): from a b = -2^31 down, the integer no longer
// fits the low word, and its wrapped value gave e^-x of x = 6e6 as -3e218.
__device__ __forceinline__ double exp2_tab(double a, double b, const double* tab) {
  constexpr double big = 6755399441055744.0;
  const double t = fma(a, b, big);
  const double f = fma(a, b, -(t - big));
  const long long d = __double_as_longlong(t) - 0x4338000000000000ll;  // the integer, where it is in range
  const int n = (int)d;
  const double p = tab[n & (EXP64_N - 1)];
  const double e = scale64(fma(p, exp64_poly(f), p), n >> 8);
  if ((unsigned long long)(d + 1021 * EXP64_N) < 2044ull * EXP64_N) return e;
  if ((__double2hiint(t) & 0x7fffffff) >= 0x7ff80000) return t;
  return __hiloint2double(d < 0 ? 0 : 0x7ff00000, 0);
}
// log2 x of a positive normal x within FP32's range: the FP32 value l, and
// log2(1 + t), t = x 2^-l - 1, |t| < 1e-6, by two terms (the third is below 1e-18)
__device__ __forceinline__ double log2_tab(double x, const double* tab) {
  const double l = f64_of(log2f(f32_of(x)));
  const double t = fma(x, exp2_tab(-EXP64_N, l, tab), -1.0);
  return fma(t * 1.442695040888963407359924681001892137, fma(-0.5, t, 1.0), l);
}
// -lambda (u - U)^2 as a 256th of a power of two: a = EXP64_LOG2E lambda
constexpr double EXP64_LOG2E = -256.0 * 1.442695040888963407359924681001892137;

// x^y of positive normal x for one y: with j = round(256 log2 x) (FP32),
// x^y = 2^(y j / 256) (1 + t)^y, t = x 2^(-j / 256) - 1 with |t| < 0.0014, five
// terms of the binomial series; 18 FP64 instructions.
struct Pow64 {
  double y, b[5];  // b[k]: binomial coefficient of t^(k+1)
};
inline Pow64 pow64_of(double y) {
  Pow64 p;
  p.y = y;
  double c = 1.0;
  for (int k = 0; k < 5; ++k) {
    c = c * (y - k) / (k + 1);
    p.b[k] = c;
  }
  return p;
}
__device__ __forceinline__ double pow_tab(double x, const Pow64& p, const double* tab) {
  const int hi = __double2hiint(x);
  const float m = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | ((unsigned)__double2loint(x) >> 29));
  const int j = ((hi >> 20) - 1023) * EXP64_N + __float2int_rn((float)EXP64_N * __log2f(m));
  const double t = fma(x, scale64(tab[-j & (EXP64_N - 1)], -j >> 8), -1.0);
  const double s = t * fma(fma(fma(fma(p.b[4], t, p.b[3]), t, p.b[2]), t, p.b[1]), t, p.b[0]);
  // (double)j: the integer in the low word of 2^52 + 2^31
  const double jd = __hiloint2double(0x43300000, j ^ 0x80000000) - 4503601774854144.0;
  double f;
  const int n = split64(p.y, jd, f);
  const double q = exp64_poly(f);
  const double e = scale64(tab[n & (EXP64_N - 1)], n >> 8);
  return fma(e, fma(q, s, q + s), e);
}

}  // namespace kb
