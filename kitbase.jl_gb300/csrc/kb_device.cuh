// kb_device.cuh -- device-side data layout and pointwise physics of the DVM step.
//
// Layout in HBM (one handle):
//   h, b   [cell][vstride] of T (double for KB_PREC_FP64, float for KB_PREC_FP32),
//          velocity index fastest (v = iu + nu*iv), vstride = nvel rounded up to 4;
//          two copies (ping-pong) because the update reads neighbour cells.
//   w, prim [cell][4] double (1D uses 3 entries), sw [cell][2][4] double.
//   per face: FaceParam (interface equilibrium, time integrals, UGKS slopes) and
//   fw [face][4] double in the global frame.
//   per cell: CellParam (new Maxwellian, collision factors, Shakhov coefficients).
// Cells are ordered x fastest with ghost layers included; x faces ((nx+1)*ny,
// i fastest) and y faces (nx*(ny+1)).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_f64.cuh"

namespace kb {

constexpr double PI = 3.141592653589793238462643383279502884;
constexpr double LOG2E = 1.442695040888963407359924681001892137;

enum { FLUX_KFVS = 0, FLUX_KCU = 1, FLUX_UGKS = 2 };
enum { COLL_BGK = 0, COLL_SHAKHOV = 1 };
enum { BC_FIX = 0, BC_EXTRA = 1, BC_PERIOD = 2, BC_MAXWELL = 3 };

// Geometry of one solve, passed by value to every kernel.
struct Geo {
  int D, NW;
  int nx, ny, ngx, ngy, nxt, nyt;
  int nu, nvel, vstride;
  int interp;  // 1 or 2
  int bc[4];
  double dx, dy, x0, y0;
  double K, gamma, mu_ref, omega, Pr;
  // K in the terms of the second distribution b (its equilibrium
  // B = H K / (2 lambda), the Shakhov factor 2 lambda c^2 + K - 5): K for the
  // 2F models, 0 for the 1F models, which carry no b (src/Solver/step_1f.jl)
  double Kb;
  int nf;  // distributions per cell: 2 (h, b) or 1 (f, held in h; b stays 0)
  int tensor;  // 2D velocity grid u[k] = u[k mod nu], v[k] = v[k - k mod nu]
  // formed once on the host (geo_consts): FP64 divisions are dear on the device
  double rdx, rdy;   // 1 / dx, 1 / dy
  double rds;        // 1 / cell size (dx, or dx dy)
  double hg;         // 0.5 / (gamma - 1)
  double rmu;        // 1 / (2 mu_ref)
  double sfac;       // 0.8 (1 - Pr)
  double rKD;        // 1 / (K + D)
  float om1f;        // omega - 1
  Pow64 tau_pow;     // lambda^(omega - 1) of the collision time
};
inline void geo_consts(Geo& g) {
  g.rdx = 1.0 / g.dx;
  g.rdy = 1.0 / g.dy;
  g.rds = 1.0 / (g.D == 1 ? g.dx : g.dx * g.dy);
  g.hg = 0.5 / (g.gamma - 1.0);
  g.rmu = 1.0 / (2.0 * g.mu_ref);
  g.sfac = 0.8 * (1.0 - g.Pr);
  g.rKD = 1.0 / (g.K + double(g.D));
  g.om1f = float(g.omega - 1.0);
  g.tau_pow = pow64_of(g.omega - 1.0);
}

// Interface quantities of one face in the face-local frame.  KFVS uses only
// `tr` and `len`; KCU adds the equilibrium part (prim, Mt[0..1], fwa); UGKS all of it.
struct FaceParam {
  double prim[4];   // rho, U_n, U_t, lambda at the interface (1D: U_t = 0)
  double Mt[5];     // time integration coefficients
  double aL[4], aR[4], aT[4];
  double fwa[4];    // analytic (equilibrium) part of fw, local frame, times len
  double len;       // face length (1 in 1D)
  double Mxi2;      // <xi^4> moment of the interface Maxwellian
  double tr[2];     // transport coefficients incl. len: Th = tr0 un h_face - tr1 un^2 sh
};

// Per-cell quantities of the FP64 update: new Maxwellian, relaxation factors,
// old Maxwellian with the Shakhov factors.
struct CellParam {
  double rho_n, U, V, l2, cB;  // new Maxwellian: rho*(lam/pi)^(D/2), U, V, EXP64_LOG2E lambda, K/(2 lambda)
  double dtau;                  // dt / tau
  double inv;                   // 1 / (1 + dt / tau)
  double o_rho_n, oU, oV, olam, ocB;  // old Maxwellian (Shakhov term)
  double s0, s1;                // 0.8 (1 - Pr) lambda^2 / rho (old) times the old heat flux
  int upd;                      // 0: copied unchanged, 1: stepped
  int coll;                     // collision model used for this cell
};

// FP32 coefficient block of one face for the velocity-owning kernels.  With
// face-frame velocity (un, ut), c2 = un^2 + ut^2 and the monomials
// m = (un, un^2, un^3, un^2 ut, un^2 c2, un ut, un c2):
//   H  = 2^(E.x + E.y un + E.z ut + E.w c2)            (interface Maxwellian)
//   fh = H (C1 m1 + ... + C7 m7) + T.x un h_f - T.y un^2 dh
//   fb = H (D1 m1 + ... + D7 m7) + T.x un b_f - T.y un^2 db
// where h_f is the upwind face value and dh the unscaled van Leer slope
// (slope * dx), T.y already divided by dx; len is folded in.  C2..C5 and
// D2..D5 depend on the upwind side (aL for un >= 0, aR otherwise).
// For a Maxwell wall face: E is the wall Maxwellian, T.x = len dt,
// T.z = K / (2 lambda_w), T.w = rot.
struct __align__(16) FaceCoef32 {
  float4 E;
  float4 T;   // T3, T4 / dx, C1, D1
  float4 G;   // C6, C7, D6, D7
  float4 Cp;  // C2..C5 for un >= 0
  float4 Dp;  // D2..D5 for un >= 0
  float4 Cm;  // C2..C5 for un < 0
  float4 Dm;  // D2..D5 for un < 0
};

// The same block in FP64, with the Maxwellian as rho (lam/pi)^(D/2), U, V and
// EXP64_LOG2E lambda (exp2_tab).
struct Quad64 {
  double x, y, z, w;
};
struct FaceCoef64 {
  Quad64 E, T, G, Cp, Dp, Cm, Dm;
};
template <typename R> struct FaceCoefOf;
template <> struct FaceCoefOf<float> { using T = FaceCoef32; };
template <> struct FaceCoefOf<double> { using T = FaceCoef64; };

// FP32 coefficients of the pointwise cell update (velocity (u, v), c2):
//   M   = 2^(EM.x + EM.y u + EM.z v + EM.w c2),  MB = M A.x
//   OH  = 2^(EO.x + EO.y u + EO.z v + EO.w c2)   (old Maxwellian, Shakhov)
//   cq  = Q.x + Q.y u + Q.z v,  tl = TL.x + TL.y u + TL.z v + TL.w c2
//   MH += cq (tl - 5) OH,  MB += cq (tl - 3) OH Q.w
//   h   = (h + div * A.w + A.y MH) * A.z
// Cells left unchanged carry A = (0, 0, 1, 0), Q = 0 and EM.x = -200.
struct __align__(16) CellCoef32 {
  float4 EM;
  float4 A;   // cB, dt/tau, 1/(1 + dt/tau), 1/ds
  float4 EO;
  float4 Q;   // Q0, Q1, Q2, old cB
  float4 TL;
};

__host__ __device__ inline int cell_index(const Geo& g, int i, int j) {
  return (j + g.ngy) * g.nxt + (i + g.ngx);
}

// Slope rule along one direction for a cell with 0-based index i (ghosts
// outside [0, n)): 0 none, 1 van Leer (reconstruct3!), 2 forward difference,
// 3 backward difference (reconstruct2! at 2D boundaries).  Follows
// reconstruct! 1D2F (src/Solver/solver_reconstruction.jl:101-153) and 2D2F
// (:475-620): 1D without ghosts leaves cells 1 and nx at zero slope; 2D uses
// one-sided slopes at i = 1 and i = nx; ghost cells keep zero h / b slopes.
__host__ __device__ inline int slope_rule(const Geo& g, int d, int i) {
  if (g.interp == 1) return 0;
  int n = d == 0 ? g.nx : g.ny;
  int ng = d == 0 ? g.ngx : g.ngy;
  if (i < 0 || i >= n) return 0;
  if (g.D == 1) {
    if (ng == 0 && (i == 0 || i == n - 1)) return 0;
    return 1;
  }
  if (i == 0) return 2;
  if (i == n - 1) return 3;
  return 1;
}

// ---------------------------------------------------------------- limiter

// vanleer (src/Reconstruction/recon_limiter.jl:17-19) with fortsign = |1|*sign(y)
template <typename R>
__device__ __forceinline__ R jsign(R y) {
  return y > R(0) ? R(1) : (y < R(0) ? R(-1) : y);
}
template <typename R>
__device__ __forceinline__ R vanleer(R sL, R sR) {
  R aL = fabs(sL), aR = fabs(sR);
  return (jsign(sL) + jsign(sR)) * aL * aR / (aL + aR + R(1.e-7));
}

// Slope of one distribution value at a cell given its neighbours.
template <typename R>
__device__ __forceinline__ R slope_of(int rule, R qm, R q0, R qp, R inv_d) {
  if (rule == 1) return vanleer((q0 - qm) * inv_d, (qp - q0) * inv_d);
  if (rule == 2) return (qp - q0) * inv_d;
  if (rule == 3) return (q0 - qm) * inv_d;
  return R(0);
}
template <>
__device__ __forceinline__ double slope_of<double>(int rule, double qm, double q0, double qp,
                                                   double d) {
  // FP64 path divides like the reference: (q0 - qm) / dx
  if (rule == 1) return vanleer((q0 - qm) / d, (qp - q0) / d);
  if (rule == 2) return (qp - q0) / d;
  if (rule == 3) return (q0 - qm) / d;
  return 0.0;
}

// ---------------------------------------------------- scalar FP64 physics

// conserve_prim!, src/Theory/theory_macro.jl:185-206, with hg = 0.5 / (gamma - 1).
template <int NW>
__device__ __forceinline__ void conserve_prim(const double* W, double hg, double* p) {
  const double r = rcp64(W[0]);
  p[0] = W[0];
  p[1] = W[1] * r;
  if (NW == 3) {
    p[2] = W[0] * hg * rcp64(fma(-0.5 * W[1], p[1], W[2]));
    p[3] = 0.0;
  } else {
    p[2] = W[2] * r;
    p[3] = W[0] * hg * rcp64(fma(-0.5, fma(W[1], p[1], W[2] * p[2]), W[3]));
  }
}

// Transcendental functions of the face and cell parameters.  FAST (the FP32
// split form, whose fluxes are FP32 anyway) evaluates them in FP32 and widens
// the result; otherwise FP64 (tab: exp64_load).  Arithmetic and the moment
// recursions stay FP64 either way.
template <bool FAST>
__device__ __forceinline__ double t_exp_neg(double x, const double* tab) {  // e^-x, x >= 0
  return FAST ? f64_of(expf(f32_of(-x))) : exp2_tab(EXP64_LOG2E, x, tab);
}
template <bool FAST>
__device__ __forceinline__ double t_erfc(double x) { return FAST ? f64_of(erfcf(f32_of(x))) : erfc(x); }
template <bool FAST>
__device__ __forceinline__ double t_sqrt(double x) { return FAST ? f64_of(sqrtf(f32_of(x))) : sqrt64(x); }

// 1 / tau of vhs_collision_time, tau = 2 mu lambda^(1 - omega) / rho
// (src/Theory/theory_relaxation.jl:28)
template <bool FAST>
__device__ __forceinline__ double vhs_rate(const Geo& g, double rho, double lam, const double* tab) {
  const double p = FAST ? f64_of(powf(f32_of(lam), g.om1f)) : pow_tab(lam, g.tau_pow, tab);
  return g.rmu * rho * p;
}

// Half-range moments of the Gaussian (gauss_moments,
// src/Theory/theory_moments.jl:10-86) of orders 0 and 1: over u > 0,
// L0 = erfc(-s) / 2 with s = sqrt(lambda) U, L1 = U L0 + e, over u < 0,
// R0 = erfc(s) / 2, R1 = U R0 - e, e = exp(-s^2) / (2 sqrt(pi lambda)).  The
// smaller of L0 and R0 is evaluated and the other is 1 less it.
// hl = 1 / (2 lambda).
template <bool FAST>
__device__ __forceinline__ void half_range(double l, double U, double hl, const double* tab, double& L0,
                                           double& L1, double& R0, double& R1) {
  const double sl = t_sqrt<FAST>(l), x = l * (U * U);
  const double e = FAST ? f64_of(0.5f * expf(f32_of(-x)) * rsqrtf(f32_of(PI * l)))
                        : exp2_tab(EXP64_LOG2E, x, tab) * (hl * sl * 0.56418958354775628695);  // 1 / sqrt(pi)
  const double a = 0.5 * t_erfc<FAST>(sl * fabs(U)), b = 1.0 - a;
  const bool up = nonneg64(U);
  L0 = up ? b : a;
  R0 = up ? a : b;
  L1 = fma(U, L0, e);
  R1 = fma(U, R0, -e);
}

// Conserved moments of u^al (slope . psi) of a Maxwellian
// (moments_conserve_slope, src/Theory/theory_moments.jl:335-369), psi =
// (1, u, [v,] (u^2 + [v^2 +] xi^2) / 2): the tangential and internal parts
// depend on the slope and the Maxwellian alone (SlopeV), so one slope's
// half- and full-range moments of several orders share them.
template <int NW>
struct SlopeV {
  double a0, a1, c, x1, x2, V0, V1, V2, v1, v2;
  // a: slope; V: tangential velocity; hl = 1 / (2 lambda); x1, x2: <xi^2>, <xi^4>
  __device__ __forceinline__ void set(const double* a, double V, double hl, double x1_, double x2_) {
    x1 = x1_;
    x2 = x2_;
    a0 = a[0];
    a1 = a[1];
    c = 0.5 * a[NW - 1];
    const double A = fma(c, x1, a0);
    if (NW == 3) {
      V0 = A;
      return;
    }
    const double a2 = a[2];
    v1 = V;
    v2 = fma(V, V, hl);
    const double v3 = fma(V, v2, 2.0 * hl * v1), v4 = fma(V, v3, 3.0 * hl * v2);
    V0 = fma(c, v2, fma(a2, v1, A));
    V1 = fma(c, v3, fma(a2, v2, A * v1));
    V2 = fma(c, v4, fma(a2, v3, A * v2));
  }
  // M: u moments of orders al .. al + 4
  __device__ __forceinline__ void get(const double* M, double* o) const {
    const double U0 = fma(a1, M[1], c * M[2]), U1 = fma(a1, M[2], c * M[3]), U2 = fma(a1, M[3], c * M[4]);
    const double s0 = fma(M[0], V0, U0);
    o[0] = s0;
    o[1] = fma(M[1], V0, U1);
    // <xi^2 ...> = x1 (s0 - c x1 M0) + c x2 M0
    double e = fma(M[2], V0, U2) + fma(x1, s0, c * fma(-x1, x1, x2) * M[0]);
    if (NW == 4) {
      o[2] = fma(M[0], V1, v1 * U0);
      e += fma(M[0], V2, v2 * U0);
    }
    o[NW - 1] = 0.5 * e;
  }
};

// pdf_slope(prim, sw, inK) (src/Theory/theory_pdf.jl:11-49).  r0 = 1 / rho,
// hl = 1 / (2 lambda), rk = 1 / (K + D), Kd = K + D.
template <int NW>
__device__ __forceinline__ void pdf_slope(const double* p, const double* s, double r0, double hl, double rk,
                                          double Kd, double* sl) {
  constexpr int E = NW - 1;  // energy slot
  const double l = p[E], U = p[1], V = NW == 4 ? p[2] : 0.0, sv = NW == 4 ? s[2] : 0.0;
  const double q2 = NW == 4 ? fma(U, U, V * V) : U * U, c = Kd * hl;
  double t = fma(s[0], q2 - c, 2.0 * s[E]);
  t = fma(-2.0 * U, s[1], t);
  if (NW == 4) t = fma(-2.0 * V, sv, t);
  const double tl = 2.0 * l * r0;
  const double se = (2.0 * l * rk) * tl * t;
  const double s1 = fma(tl, fma(-U, s[0], s[1]), -U * se);
  double z = fma(s[0], r0, -U * s1);
  if (NW == 4) {
    const double s2 = fma(tl, fma(-V, s[0], sv), -V * se);
    z = fma(-V, s2, z);
    sl[2] = s2;
  }
  sl[0] = fma(-0.5 * (q2 + c), se, z);
  sl[1] = s1;
  sl[E] = se;
  if (NW == 3) sl[3] = 0.0;
}

// ------------------------------------------- compensated FP32 accumulation

// Packed FP32 pair arithmetic: one instruction for two values.
__device__ __forceinline__ float2 p2add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p2mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 p2fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 p2sub(float2 a, float2 b) {
  unsigned long long A = *reinterpret_cast<unsigned long long*>(&a);
  unsigned long long B = *reinterpret_cast<unsigned long long*>(&b), C;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(C) : "l"(A), "l"(B));
  return *reinterpret_cast<float2*>(&C);
}
__device__ __forceinline__ float2 p2s(float x) { return make_float2(x, x); }

// Double-float accumulator: (hi, lo) with |lo| <= ulp(hi)/2 after each add.
// Knuth's TwoSum makes every addition error-free, so the pair carries about
// 44 significant bits; it is converted exactly to FP64 (hi + lo) before the
// FP64 combination across threads.
struct DF {
  float hi, lo;
};
__device__ __forceinline__ void df_add(DF& a, float x) {
  float s = a.hi + x;
  float bp = s - a.hi;
  float e = (a.hi - (s - bp)) + (x - bp);
  a.hi = s;
  a.lo += e;
}
// df_add of two independent sums at once
__device__ __forceinline__ void p2df_add(float2& hi, float2& lo, float2 x) {
  const float2 s = p2add(hi, x);
  const float2 bp = p2sub(s, hi);
  lo = p2add(lo, p2add(p2sub(hi, p2sub(s, bp)), p2sub(x, bp)));
  hi = s;
}
__device__ __forceinline__ DF df_merge(DF a, DF b) {
  float s = a.hi + b.hi;
  float bp = s - a.hi;
  float e = (a.hi - (s - bp)) + (b.hi - bp);
  e += a.lo + b.lo;
  float hi = s + e;
  float lo = e - (hi - s);
  DF r;
  r.hi = hi;
  r.lo = lo;
  return r;
}
__device__ __forceinline__ DF df_shfl_xor(DF a, int m) {
  DF r;
  r.hi = __shfl_xor_sync(0xffffffffu, a.hi, m);
  r.lo = __shfl_xor_sync(0xffffffffu, a.lo, m);
  return r;
}

// Sums of N values over the warp (N a power of two, at most 32): a
// reduce-scatter whose first log2 N levels halve the number of values a lane
// carries, then plain levels: N - 1 + 5 - log2 N additions instead of 5 N.
// Lane l returns the total of value l >> (5 - log2 N), in a fixed order.
__device__ __forceinline__ double join(double a, double b) { return a + b; }
__device__ __forceinline__ DF join(DF a, DF b) { return df_merge(a, b); }
__device__ __forceinline__ double shfl_xor_of(double a, int m) { return __shfl_xor_sync(0xffffffffu, a, m); }
__device__ __forceinline__ DF shfl_xor_of(DF a, int m) { return df_shfl_xor(a, m); }
template <int N, typename T>
__device__ __forceinline__ T warp_sums(T* x, int lane) {
#pragma unroll
  for (int m = 16, n = N; m >= 1; m >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & m;  // the upper lanes keep the upper half
#pragma unroll
      for (int k = 0; k < n; ++k) {
        const T keep = up ? x[n + k] : x[k], give = up ? x[k] : x[n + k];
        x[k] = join(keep, shfl_xor_of(give, m));
      }
    } else {
      x[0] = join(x[0], shfl_xor_of(x[0], m));
    }
  }
  return x[0];
}
__device__ __forceinline__ double f64_total(double x) { return x; }
__device__ __forceinline__ double f64_total(DF x) { return f64_of(x.hi) + f64_of(x.lo); }

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
  return x;
}

// Accumulator selected by the storage type: FP64 path sums in double, FP32
// path in compensated double-float.
template <typename R>
struct Acc;
template <>
struct Acc<double> {
  double s;
  __device__ __forceinline__ Acc() : s(0.0) {}
  __device__ __forceinline__ void add(double x) { s += x; }
};
template <>
struct Acc<float> {
  DF s;
  __device__ __forceinline__ Acc() { s.hi = 0.f; s.lo = 0.f; }
  __device__ __forceinline__ void add(float x) { df_add(s, x); }
};

// exp of a Maxwellian exponent
__device__ __forceinline__ double mexp(double x) { return exp(x); }
__device__ __forceinline__ float mexp(float x) { return exp2f(x * float(LOG2E)); }

}  // namespace kb
