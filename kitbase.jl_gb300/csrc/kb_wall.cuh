// kb_wall.cuh -- Maxwell wall faces: the wall density and the wall's flux, one
// CTA per face (kb_kernels.cu and, beside the moment passes, kb_march.cuh).
#pragma once

#include "kb_kernels.cuh"
#include "kb_flux.cuh"
#include "kb_tma.cuh"

namespace kb {

// log2-form exponent of rho (lam/pi)^(D/2) exp(-lam ((un-U)^2 + (ut-V)^2)) as
// E.x + E.y un + E.z ut + E.w c2; the log2 of the density factor in FP32, or (tab)
// in FP64: a wall's Maxwellian is rounded to FP32 once.
__device__ __forceinline__ float4 maxwell_exp2(double rho_n, double U, double V, double lam,
                                               const double* tab = nullptr) {
  float4 E;
  const float rf = f32_of(rho_n);
  const double ll = lam * LOG2E, lU = ll * U, lV = ll * V;
  E.x = rf > 0.f ? f32_of((tab ? log2_tab(rho_n, tab) : f64_of(log2f(rf))) - fma(lU, U, lV * V)) : -200.f;
  E.y = f32_of(lU + lU);
  E.z = f32_of(lV + lV);
  E.w = f32_of(-ll);
  return E;
}

// One coefficient in the block's precision.
__device__ __forceinline__ void put(float& o, double x) { o = f32_of(x); }
__device__ __forceinline__ void put(double& o, double x) { o = x; }
__device__ __forceinline__ void put_maxwell(float4& E, double rho_n, double U, double V, double lam) {
  E = maxwell_exp2(rho_n, U, V, lam);
}
__device__ __forceinline__ void put_maxwell(Quad64& E, double rho_n, double U, double V, double lam) {
  E.x = rho_n;
  E.y = U;
  E.z = V;
  E.w = EXP64_LOG2E * lam;
}

// flux_boundary_maxwell! 1D2F1V (src/Flux/flux_boundary.jl:39-61) and 2D2F2V
// (:190-220) in the face-local frame; rot = +1 on the left / bottom wall and
// -1 on the right / top wall (src/Solver/evolve_boundary.jl).  One CTA of
// WALL_T threads per wall face (DevState::wall_list): the velocities are
// shared by all its warps, each warp sums its part, and thread 0 adds the
// warps' sums in warp order (deterministic) and finishes the face.
constexpr int WALL_T = 128;
// exp(-lw e) from lw scaled to the base-two exponent of each form
__device__ __forceinline__ float wall_exp(float l2, float e, const double*) { return exp2f(l2 * e); }
__device__ __forceinline__ double wall_exp(double l2, double e, const double* tab) { return exp2_tab(l2, e, tab); }
// Block b of the wall faces (of a grouped launch: of all members').  The CTA may
// have more than WALL_T threads; the others only meet the barrier.
template <typename R, int D, bool GRP = false>
__device__ __forceinline__ void wall_face(const DevState& sp, double dt_arg, int b) {
  __shared__ double part[WALL_T / 32][8];
  const double* tab = EXP64_TAB;
  int lb;
  const int gr = group_member<GRP, GK_WALL>(sp, lb, b);
  KB_GROUP_STATE(GRP, sp, gr);
  const double dt = GRP ? sp.grp->dt[gr] : dt_arg;
  const Geo& g = s.g;
  const int f = s.wall_list[lb];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  FaceGeo r = face_geo(g, f);
  int pos = r.d == 0 ? r.fi : r.fj;
  int rot = pos == 0 ? 1 : -1;
  int c = pos == 0 ? r.cR : r.cL;  // the interior cell next to the wall
  const double* wp = s.wall + (long)f * 4;
  double bw[4];
  if (D == 1) {
    bw[0] = wp[0]; bw[1] = wp[1]; bw[2] = 0.0; bw[3] = wp[2];
  } else if (r.d == 0) {
    bw[0] = wp[0]; bw[1] = wp[1]; bw[2] = wp[2]; bw[3] = wp[3];
  } else {
    bw[0] = wp[0]; bw[1] = wp[2]; bw[2] = -wp[1]; bw[3] = wp[3];
  }
  double lw = bw[3];
  const R* H = (const R*)s.h[s.cur];
  const R* Bq = (const R*)s.b[s.cur];
  const R* U = vtab<R>(s, 0);
  const R* V = vtab<R>(s, 1);
  const R* W = vtab<R>(s, 2);
  long vs = g.vstride;
  R Uw = R(bw[1]), Vw = R(bw[2]);
  // One pass: the outgoing half from the interior cell's h, b; the incoming
  // half as moments of the unit-density wall Maxwellian, scaled by the wall
  // density afterwards in FP64.  The mass flux S0 = SF + rho_n * I0 then
  // cancels to FP64 round-off by construction (the density is chosen so that
  // no mass crosses the wall), also when h is stored in FP32.
  Acc<R> o0, o1, o2, o3, i0, i1, i2, i3;
  const R Lw2 = R(lw * (sizeof(R) == 8 ? EXP64_LOG2E : -LOG2E));
  for (int v = threadIdx.x < WALL_T ? threadIdx.x : g.nvel; v < g.nvel; v += WALL_T) {
    R un, ut;
    if (D == 1) { un = U[v]; ut = R(0); }
    else if (r.d == 0) { un = U[v]; ut = V[v]; }
    else { un = V[v]; ut = -U[v]; }
    const bool in = rot > 0 ? !(un < R(0)) : !(un > R(0));
    R c2 = un * un;
    if (D == 2) c2 += ut * ut;
    if (in) {
      R du = un - Uw, e = du * du;
      if (D == 2) { R dv = ut - Vw; e += dv * dv; }
      const R t = W[v] * un * wall_exp(Lw2, e, tab);
      i0.add(t);
      i1.add(t * un);
      if (D == 2) i2.add(t * ut);
      i3.add(t * c2);
    } else {
      const R t = W[v] * un * H[(long)c * vs + v];
      o0.add(t);
      o1.add(t * un);
      if (D == 2) o2.add(t * ut);
      o3.add(t * c2 + W[v] * un * Bq[(long)c * vs + v]);
    }
  }
  {
    decltype(o0.s) x[8] = {o0.s, o1.s, o2.s, o3.s, i0.s, i1.s, i2.s, i3.s};
    const double t = f64_total(warp_sums<8>(x, lane));
    if ((lane & 3) == 0 && wid < WALL_T / 32) part[wid][lane >> 2] = t;
  }
  __syncthreads();
  // lane k of the first warp adds the warps' sums k in warp order
  if (wid != 0) return;
  double Tk = part[0][lane & 7];
  for (int w = 1; w < WALL_T / 32; ++w) Tk += part[w][lane & 7];
  double T[8];
  for (int k = 0; k < 8; ++k) T[k] = __shfl_sync(0xffffffffu, Tk, k);
  if (lane != 0) return;
  const double norm = D == 1 ? sqrt64(lw * (1.0 / PI)) : lw * (1.0 / PI);
  const double SF = T[0], I0 = T[4];
  const double rn = -SF * rcp64(I0);  // wall density times the Maxwellian's normalisation
  const double rho = rn * rcp64(norm);
  const double cBw = g.Kb * (0.5 * rcp64(lw));
  double len = D == 2 ? (r.d == 0 ? g.dy : g.dx) : 1.0;
  double sc = D == 2 ? len * dt : dt;
  const double S0 = SF + rn * I0;
  const double S1 = T[1] + rn * T[5];
  const double S2 = D == 2 ? T[2] + rn * T[6] : 0.0;
  const double S3 = T[3] + rn * (T[7] + cBw * I0);
  s.rhow[f] = rho;
  if (sizeof(R) == 4) {
    FaceCoef32 wc;
    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    wc.G = wc.Cp = wc.Dp = wc.Cm = wc.Dm = z;
    wc.E = maxwell_exp2(rn, bw[1], bw[2], lw, tab);
    wc.T = make_float4(f32_of(sc), 0.f, f32_of(cBw), rot > 0 ? 1.f : -1.f);
    s.fc[f] = wc;
  } else {
    FaceCoef64 wc{};
    put_maxwell(wc.E, rn, bw[1], bw[2], lw);
    wc.T.x = sc;
    wc.T.z = cBw;
    wc.T.w = rot > 0 ? 1.0 : -1.0;
    s.fc64[f] = wc;
  }
  double fl[4] = {S0 * sc, S1 * sc, 0.0, 0.0};
  if (D == 1) {
    fl[2] = 0.5 * S3 * sc;
  } else {
    fl[2] = S2 * sc;
    fl[3] = 0.5 * S3 * sc;
  }
  double* out = s.fw + (long)f * 4;
  if (D == 2 && r.d == 1) {
    out[0] = fl[0]; out[1] = -fl[2]; out[2] = fl[1]; out[3] = fl[3];
  } else {
    for (int k = 0; k < 4; ++k) out[k] = fl[k];
  }
}

}  // namespace kb
