// kb_kernels.cu -- sm_103a kernels of the DVM time step (1D2F1V, 2D2F2V).
//
// One step is: [w slopes] -> [face parameters] -> face moments (fw) ->
// [Maxwell walls] -> [Shakhov heat flux] -> cell parameters (w, prim, tau,
// residual partials) -> pointwise update of h, b -> [ghost fill] -> residual.
// The pointwise face fluxes fh, fb are never stored: the update kernel forms
// them again from the neighbour cells, so h and b are read from HBM and
// written once per step apart from stencil re-reads that hit L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>
#include <stdio.h>

#include "kb_kernels.cuh"
#include "kb_flux.cuh"
#include "kb_tma.cuh"
#include "kb_wall.cuh"

namespace kb {

// Classification of every face (0 not computed, 1 interior flux, 2 Maxwell wall):
// evolve! computes faces idx0:idx1 (all faces when ghosts exist, interior
// faces otherwise; src/Solver/solver_evolution.jl:64-89, :608-679) and
// evolve_boundary! replaces the wall faces (src/Solver/evolve_boundary.jl).
void face_kinds_host(const Geo& g, signed char* kind) {
  int n = face_count(g);
  for (int f = 0; f < n; ++f) {
    FaceGeo r = face_geo(g, f);
    int pos = r.d == 0 ? r.fi : r.fj;
    int nn = r.d == 0 ? g.nx : g.ny;
    int ng = r.d == 0 ? g.ngx : g.ngy;
    signed char k = 1;
    if ((pos == 0 || pos == nn) && ng == 0) k = 0;
    int side = r.d == 0 ? (pos == 0 ? 0 : (pos == nn ? 1 : -1)) : (pos == 0 ? 2 : (pos == nn ? 3 : -1));
    if (side >= 0 && g.bc[side] == BC_MAXWELL) k = 2;
    kind[f] = k;
  }
}

// ------------------------------------------------------------ w slopes

// reconstruct! for w (src/Solver/solver_reconstruction.jl:111-122 1D, :496-537 2D):
// one thread per (physical cell, direction).
template <bool GRP = false>
__global__ void k_wslope(DevState sp) {
  pdl_wait();
  pdl_next();
  int lb;
  const int gr = group_member<GRP, GK_WSLOPE>(sp, lb);
  KB_GROUP_STATE(GRP, sp, gr);
  const Geo& g = s.g;
  int t = lb * blockDim.x + threadIdx.x;
  int n = g.nx * g.ny;
  if (t >= n * g.D) return;
  int d = t / n, c0 = t % n;
  int i = c0 % g.nx, j = c0 / g.nx;
  int c = cell_index(g, i, j);
  int rule = slope_rule(g, d, d == 0 ? i : j);
  int step = d == 0 ? 1 : g.nxt;
  // dx = 0.5 * (dx[i-1] + dx[i]) on a uniform mesh
  double* out = s.sw + ((long)c * 2 + d) * 4;
  const double rd = d == 0 ? g.rdx : g.rdy;
  const double eps = 1.e-7 * (d == 0 ? g.dx : g.dy);
  for (int k = 0; k < g.NW; ++k) {
    double q0 = s.w[(long)c * 4 + k];
    double qm = (rule == 1 || rule == 3) ? s.w[(long)(c - step) * 4 + k] : 0.0;
    double qp = (rule == 1 || rule == 2) ? s.w[(long)(c + step) * 4 + k] : 0.0;
    out[k] = rd * (rule == 1 ? vl64(qm, q0, qp, eps) : (rule == 2 ? qp - q0 : (rule == 3 ? q0 - qm : 0.0)));
  }
}

// ------------------------------------------------------- face parameters

// Monomial coefficients of the interface flux (see FaceCoef32, FaceCoef64); rdd
// = 1 / cell size along the normal, hl = 1 / (2 lambda).
template <int D, int FLUX, typename FC>
__device__ __forceinline__ void face_coef(FC& c, const Geo& g, const FaceParam& P, double rdd, double hl) {
  constexpr bool FAST = sizeof(c.E.x) == 4;
  c = FC{};
  put(c.T.x, P.tr[0]);
  put(c.T.y, P.tr[1] * rdd);
  if (FLUX == FLUX_KFVS) return;
  const double lam = P.prim[3], rho = P.prim[0], len = P.len;
  const double rho_n = D == 1 ? rho * t_sqrt<FAST>(lam * (1.0 / PI)) : rho * (lam * (1.0 / PI));
  put_maxwell(c.E, rho_n, P.prim[1], P.prim[2], lam);
  const double cB = g.Kb * hl, M0 = P.Mt[0] * len;
  if (FLUX == FLUX_KCU) {
    put(c.T.z, M0);
    put(c.T.w, M0 * cB);
    return;
  }
  const double* t = P.aT;
  const double M1 = P.Mt[1] * len, M2 = P.Mt[2] * len, M1B = M1 * cB, M2B = M2 * cB, X2 = P.Mxi2;
  const double te = 0.5 * t[D + 1];
  put(c.T.z, fma(M2, fma(te, cB, t[0]), M0));
  put(c.T.w, fma(M0, cB, fma(M2B, t[0], M2 * te * X2)));
  if (D == 2) {
    put(c.G.x, M2 * t[2]);
    put(c.G.z, M2B * t[2]);
  }
  put(c.G.y, M2 * te);
  put(c.G.w, M2B * te);
  const double M2t = M2 * t[1], M2Bt = M2B * t[1];
  // one upwind side's slope terms (a = aL for un >= 0, aR otherwise)
  auto side = [&](const double (&a)[4], auto& C, auto& Dd) {
    const double ae = 0.5 * a[D + 1];
    put(C.x, fma(M1, fma(ae, cB, a[0]), M2t));
    put(C.y, M1 * a[1]);
    if (D == 2) put(C.z, M1 * a[2]);
    put(C.w, M1 * ae);
    put(Dd.x, fma(M1B, a[0], fma(M1 * ae, X2, M2Bt)));
    put(Dd.y, M1B * a[1]);
    if (D == 2) put(Dd.z, M1B * a[2]);
    put(Dd.w, M1B * ae);
  };
  side(P.aL, c.Cp, c.Dp);
  side(P.aR, c.Cm, c.Dm);
}

// Interface equilibrium from the two half Maxwellians (flux_kcu.jl:480-495,
// flux_ugks.jl:47-56), then the KCU / UGKS time integrals, UGKS slopes and
// the analytic part of fw.  One thread per face.
// FAST: the FP32 split form (transcendentals in FP32, see t_exp_neg).
// Bound by the FP64 pipe: about 320 (UGKS) or 110 (KCU) FP64 instructions per
// face where moment by moment evaluation with divisions took 800 and 300.
template <int D, int FLUX, bool FAST, bool GRP = false>
__global__ void k_face_param(DevState sp, double dt_arg) {
  __shared__ double tab[FAST || FLUX == FLUX_KFVS ? 1 : EXP64_N];
  if (!FAST && FLUX != FLUX_KFVS) {
    exp64_load(tab, threadIdx.x, blockDim.x);
    __syncthreads();
  }
  pdl_wait();
  pdl_next();
  int lb;
  const int gr = group_member<GRP, GK_FACE>(sp, lb);
  KB_GROUP_STATE(GRP, sp, gr);
  const double dt = GRP ? sp.grp->dt[gr] : dt_arg;
  const Geo& g = s.g;
  int f = lb * blockDim.x + threadIdx.x;
  if (f >= s.nface_x + s.nface_y) return;
  if (s.kind[f] != 1) return;
  FaceGeo r = face_geo(g, f);
  constexpr int NW = D + 2, E = D + 1;
  const double dxh = 0.5 * (r.d == 0 ? g.dx : g.dy), rdd = r.d == 0 ? g.rdx : g.rdy;
  const double len = D == 1 ? 1.0 : face_len(g, r.d, r.fi, r.fj);
  FaceParam P;
  for (int k = 0; k < 4; ++k) {
    P.prim[k] = 0;
    P.aL[k] = P.aR[k] = P.aT[k] = P.fwa[k] = 0;
  }
  for (int k = 0; k < 5; ++k) P.Mt[k] = 0;
  P.len = len;
  P.Mxi2 = 0;
  P.tr[0] = P.tr[1] = 0;
  double hl = 0.0;
  if (FLUX == FLUX_KFVS) {
    P.tr[0] = dt * len;
    P.tr[1] = 0.5 * (dt * dt) * len;
  } else {
    // face states of w (local frame): w + dx/2 sw from the left, w - dx/2 sw from the right
    double wl[4], wr[4], wL[4], wR[4];
    const double* sl = s.sw + ((long)r.cL * 2 + r.d) * 4;
    const double* sr = s.sw + ((long)r.cR * 2 + r.d) * 4;
    for (int k = 0; k < 4; ++k) {
      wl[k] = k < NW ? fma(dxh, sl[k], s.w[(long)r.cL * 4 + k]) : 0.0;
      wr[k] = k < NW ? fma(-dxh, sr[k], s.w[(long)r.cR * 4 + k]) : 0.0;
    }
    if (NW == 4 && r.d == 1) {  // local_frame with n = (0, 1)
      wL[0] = wl[0]; wL[1] = wl[2]; wL[2] = -wl[1]; wL[3] = wl[3];
      wR[0] = wr[0]; wR[1] = wr[2]; wR[2] = -wr[1]; wR[3] = wr[3];
    } else {
      for (int k = 0; k < 4; ++k) { wL[k] = wl[k]; wR[k] = wr[k]; }
    }
    double wi[4] = {0.0, 0.0, 0.0, 0.0}, p[4], pj = 0.0, ps = 0.0;  // pj, ps: pressure jump and sum (KCU)
    // the half of one side's Maxwellian that crosses the face (its conserved moments)
    auto half = [&](const double* w, bool left) {
      double q[4], L0, L1, R0, R1;
      conserve_prim<NW>(w, g.hg, q);
      const double h = 0.5 * rcp64(q[E]);
      half_range<FAST>(q[E], q[1], h, tab, L0, L1, R0, R1);
      const double m0 = q[0] * (left ? L0 : R0), m1 = q[0] * (left ? L1 : R1);
      const double V = NW == 4 ? q[2] : 0.0;
      wi[0] += m0;
      wi[1] += m1;
      if (NW == 4) wi[2] = fma(m0, V, wi[2]);
      // <u^2> + <v^2> + <xi^2>
      const double t = NW == 4 ? fma(V, V, h + g.K * h) : g.K * h;
      wi[E] = fma(0.5, fma(q[1], m1, fma(h, m0, m0 * t)), wi[E]);
      if (FLUX == FLUX_KCU) {
        const double pr = q[0] * h;  // pressure: rho / (2 lambda)
        pj = left ? pr : pj - pr;
        ps += pr;
      }
    };
    half(wL, true);
    half(wR, false);
    conserve_prim<NW>(wi, g.hg, p);
    const double lam = p[E], U = p[1], V = NW == 4 ? p[2] : 0.0;
    hl = 0.5 * rcp64(lam);
    P.prim[0] = p[0];
    P.prim[1] = U;
    P.prim[2] = V;
    P.prim[3] = lam;
    const double itau = vhs_rate<FAST>(g, p[0], lam, tab);
    const double x1 = g.K * hl, x2 = fma(2.0 * hl, x1, x1 * x1);  // <xi^2>, <xi^4>
    const double v2 = NW == 4 ? fma(V, V, hl) : 0.0;
    double Mu[7];
    Mu[0] = 1.0;
    Mu[1] = U;
    Mu[2] = fma(U, U, hl);
    Mu[3] = fma(U, Mu[2], 2.0 * hl * U);
    // u times the conserved moments of the interface Maxwellian
    double Muv[4] = {Mu[1], Mu[2], 0.0, 0.0};
    if (NW == 4) Muv[2] = Mu[1] * V;
    Muv[E] = 0.5 * fma(Mu[1], v2 + x1, Mu[3]);
    if (FLUX == FLUX_KCU) {
      const double tau = rcp64(itau) + fabs(pj) * rcp64(ps) * (2.0 * dt);
      P.Mt[1] = tau * (1.0 - t_exp_neg<FAST>(dt * rcp64(tau), tab));
      P.Mt[0] = dt - P.Mt[1];
      const double m = P.Mt[0] * p[0] * len;
      for (int k = 0; k < NW; ++k) P.fwa[k] = m * Muv[k];
      P.tr[0] = P.Mt[1] * len;
    } else {
      const double tau = rcp64(itau), rh = 2.0 * rdd, r0 = rcp64(p[0]), Kd = g.K + double(D), rk = g.rKD;
      double dL[4] = {0.0, 0.0, 0.0, 0.0}, dR[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = 0; k < NW; ++k) {
        dL[k] = (wi[k] - wL[k]) * rh;
        dR[k] = (wR[k] - wi[k]) * rh;
      }
      pdf_slope<NW>(p, dL, r0, hl, rk, Kd, P.aL);
      pdf_slope<NW>(p, dR, r0, hl, rk, Kd, P.aR);
      double ML[7], MR[7];
      half_range<FAST>(lam, U, hl, tab, ML[0], ML[1], MR[0], MR[1]);
      for (int i = 2; i <= 6; ++i) {
        const double q = double(i - 1) * hl;
        if (i > 3) Mu[i] = fma(U, Mu[i - 1], q * Mu[i - 2]);
        ML[i] = fma(U, ML[i - 1], q * ML[i - 2]);
        MR[i] = Mu[i] - ML[i];
      }
      SlopeV<NW> sL, sR, sT;
      sL.set(P.aL, V, hl, x1, x2);
      sR.set(P.aR, V, hl, x1, x2);
      double a[4], b[4], tmp[4] = {0.0, 0.0, 0.0, 0.0};
      sL.get(ML + 1, a);
      sR.get(MR + 1, b);
      for (int k = 0; k < NW; ++k) tmp[k] = -p[0] * (a[k] + b[k]);
      pdf_slope<NW>(p, tmp, r0, hl, rk, Kd, P.aT);
      const double ex = t_exp_neg<FAST>(dt * itau, tab);
      P.Mt[3] = tau * (1.0 - ex);
      P.Mt[4] = fma(-tau * dt, ex, tau * P.Mt[3]);
      P.Mt[0] = dt - P.Mt[3];
      P.Mt[1] = fma(-tau, P.Mt[0], P.Mt[4]);
      P.Mt[2] = fma(-tau, P.Mt[0], 0.5 * (dt * dt));
      sT.set(P.aT, V, hl, x1, x2);
      double c[4];
      sL.get(ML + 2, a);
      sR.get(MR + 2, b);
      sT.get(Mu + 1, c);
      const double m = p[0] * len, m0 = m * P.Mt[0], m1 = m * P.Mt[1], m2 = m * P.Mt[2];
      for (int k = 0; k < NW; ++k) P.fwa[k] = fma(m0, Muv[k], fma(m1, a[k] + b[k], m2 * c[k]));
      P.Mxi2 = x2;
      P.tr[0] = P.Mt[3] * len;
      P.tr[1] = P.Mt[4] * len;
    }
  }
  s.fp[f] = P;
  if constexpr (FAST) face_coef<D, FLUX>(s.fc[f], g, P, rdd, hl);
  else face_coef<D, FLUX>(s.fc64[f], g, P, rdd, hl);
}

// ------------------------------------------------------------ Maxwell walls

// The wall faces by themselves (the stages of a step one by one); a whole step
// takes them in the moment passes' launch.
template <typename R, int D>
__global__ void __launch_bounds__(WALL_T) k_wall(DevState s, double dt) {
  pdl_wait();
  pdl_next();
  wall_face<R, D>(s, dt, blockIdx.x);
}

// ------------------------------------------------------- cell parameters

// Update group of a physical cell: 0 fixed (copied), 1 interior, 2 boundary
// (update! loops 2:nx-1 / 2:nx-1 x 2:ny-1, update_boundary! the rest when the
// side is not :fix; src/Solver/solver_update.jl, update_boundary.jl).
__device__ inline int update_group(const Geo& g, int i, int j) {
  if (g.D == 1) {
    if (i >= 1 && i <= g.nx - 2) return 1;
    if (i == 0 && g.bc[0] != BC_FIX) return 2;
    if (i == g.nx - 1 && g.bc[1] != BC_FIX) return 2;
    return 0;
  }
  if (i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2) return 1;
  if (i == 0) return g.bc[0] != BC_FIX ? 2 : 0;
  if (i == g.nx - 1) return g.bc[1] != BC_FIX ? 2 : 0;
  if (j == 0) return g.bc[2] != BC_FIX ? 2 : 0;
  return g.bc[3] != BC_FIX ? 2 : 0;
}

// step! scalar part (src/Solver/step_2f.jl:6-64, :179-249): Shakhov factors of
// the old state, w += flux divergence, prim, tau.  One thread per physical
// cell; res: each block writes its residual partials in a fixed order.  FAST
// (the FP32 split form): tau and the exponent offsets of the coefficient
// blocks with FP32 transcendentals; w and prim stay FP64.  BS threads per
// block (32 on small grids, 256 otherwise: DevState::cell_bs).  Bound by the
// FP64 pipe and, on small grids, by its latency: about 55 FP64 instructions a
// cell (FP32 split, BGK) where divisions, conversions and the unused form's
// coefficients took 350.
template <int D, bool FAST, int BS, bool GRP = false>
__global__ void __launch_bounds__(BS) k_cell_param(DevState sp, double dt_arg, int res) {
  __shared__ double tab[FAST ? 1 : EXP64_N];
  if (!FAST) {
    exp64_load(tab, threadIdx.x, BS);
    __syncthreads();
  }
  pdl_wait();
  pdl_next();
  int lb;
  const int gr = group_member<GRP, GK_CELL>(sp, lb);
  KB_GROUP_STATE(GRP, sp, gr);
  const double dt = GRP ? sp.grp->dt[gr] : dt_arg;
  const Geo& g = s.g;
  __shared__ double red[BS / 32][16];
  int t = lb * BS + threadIdx.x;
  double rr[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int grp = 0;
  if (t < g.nx * g.ny) {
    int i = t % g.nx, j = t / g.nx;
    int c = cell_index(g, i, j);
    grp = update_group(g, i, j);
    constexpr int NW = D + 2;  // compile-time, so the small arrays stay in registers
    const int coll = (D == 1 && grp == 2) ? COLL_BGK : s.coll;
    const bool shak = grp && coll == COLL_SHAKHOV;
    double* w = s.w + (long)c * 4;
    double* p = s.prim + (long)c * 4;
    double po[4] = {1.0, 0.0, 0.0, 1.0}, q0 = 0.0, q1 = 0.0;
    if (shak) {
      for (int k = 0; k < NW; ++k) po[k] = p[k];
      q0 = s.q[(long)c * 2 + 0];
      q1 = D == 2 ? s.q[(long)c * 2 + 1] : 0.0;
    }
    double pn[4] = {0.0, 0.0, 0.0, 0.0}, rho_n = 0.0, cB = 0.0, dtau = 0.0, inv = 1.0;
    if (grp) {
      double wn[4];
      const int fx = j * (g.nx + 1) + i;
      const double* fL = s.fw + (long)fx * 4;
      const double* fR = s.fw + (long)(fx + 1) * 4;
      const int fy = D == 2 ? s.nface_x + j * g.nx + i : 0;
      const double* fD = s.fw + (long)fy * 4;
      const double* fU = s.fw + (long)(fy + g.nx) * 4;
      for (int k = 0; k < NW; ++k) {
        double d = fL[k] - fR[k];
        if (D == 2) d = d + fD[k] - fU[k];
        const double wo = w[k];
        wn[k] = fma(d, g.rds, wo);
        w[k] = wn[k];
        if (res) {
          const double dw = wn[k] - wo;
          rr[k] = dw * dw;
          rr[4 + k] = fabs(wn[k]);
        }
      }
      conserve_prim<NW>(wn, g.hg, pn);
      for (int k = 0; k < NW; ++k) p[k] = pn[k];
      const double lam = pn[NW - 1];
      const double lp = lam * (1.0 / PI);
      rho_n = D == 1 ? pn[0] * t_sqrt<FAST>(lp) : pn[0] * lp;
      cB = g.Kb * (0.5 * rcp64(lam));
      dtau = dt * vhs_rate<FAST>(g, pn[0], lam, tab);
      inv = rcp64(1.0 + dtau);
      if (!pos64(pn[0]) || !pos64(lam) || !isfinite(f32_of(pn[1]))) atomicOr(s.status, 1);
    }
    const double lo = po[NW - 1], lop = lo * (1.0 / PI), oV = D == 2 ? po[2] : 0.0;
    double o_rho_n = 0.0, ocB = 0.0, s0 = 0.0, s1 = 0.0;
    if (shak) {
      o_rho_n = D == 1 ? po[0] * t_sqrt<FAST>(lop) : po[0] * lop;
      ocB = g.Kb * (0.5 * rcp64(lo));
      const double sf = g.sfac * (lo * lo) * rcp64(po[0]);
      s0 = sf * q0;
      s1 = sf * q1;
    }
    const double lam = pn[NW - 1], V = D == 2 ? pn[2] : 0.0;
    if (FAST) {
      CellCoef32 K;
      float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      K.EM = K.EO = K.Q = K.TL = z;
      K.EM.x = K.EO.x = -200.f;
      K.A = make_float4(0.f, 0.f, 1.f, 0.f);
      if (grp) {
        K.EM = maxwell_exp2(rho_n, pn[1], V, lam);
        K.A = make_float4(f32_of(cB), f32_of(dtau), f32_of(inv), f32_of(g.rds));
        if (shak) {
          K.EO = maxwell_exp2(o_rho_n, po[1], oV, lo);
          K.Q = make_float4(f32_of(-fma(s0, po[1], s1 * oV)), f32_of(s0), f32_of(s1), f32_of(ocB));
          const double l2 = 2.0 * lo, lU = l2 * po[1], lV = l2 * oV;
          K.TL = make_float4(f32_of(fma(lU, po[1], fma(lV, oV, g.Kb))), f32_of(-2.0 * lU), f32_of(-2.0 * lV),
                             f32_of(l2));
        }
      }
      s.cc[c] = K;
    } else {
      CellParam P;
      P.upd = grp ? 1 : 0;
      P.coll = coll;
      P.rho_n = rho_n;
      P.U = pn[1];
      P.V = V;
      P.l2 = EXP64_LOG2E * lam;
      P.cB = cB;
      P.dtau = dtau;
      P.inv = inv;
      P.o_rho_n = o_rho_n;
      P.oU = po[1];
      P.oV = oV;
      P.olam = lo;
      P.ocB = ocB;
      P.s0 = s0;
      P.s1 = s1;
      s.cp[c] = P;
    }
  }
  if (!res) return;  // uniform over the launch
  // deterministic block partials: interior (grp 1) and boundary (grp 2) sums
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double x[16];
  for (int k = 0; k < 8; ++k) {
    x[k] = grp == 1 ? rr[k] : 0.0;
    x[8 + k] = grp == 2 ? rr[k] : 0.0;
  }
  const double sum = warp_sums<16>(x, lane);
  if ((lane & 1) == 0) red[wid][lane >> 1] = sum;
  __syncthreads();
  if (threadIdx.x < 16) {
    double a = red[0][threadIdx.x];
    for (int k = 1; k < BS / 32; ++k) a += red[k][threadIdx.x];
    s.blockres[(long)lb * 16 + threadIdx.x] = a;
  }
}

// ---------------------------------------------- Maxwellians on product grids

// FP64: where the velocity grid is a product of nu and nv abscissae, so is a
// Maxwellian, and the update takes its value as one product of two entries
// instead of some 12 FP64 instructions for the exponential and its argument.
// One thread per face or cell and abscissa; a cell's old Maxwellian (Shakhov)
// follows its new one.  128^2 cells x 32^2 velocities, UGKS
// and BGK: this kernel 71 us, the update 5,205 -> 3,989; 64^2 x 28^2, KCU and
// Shakhov, walls: 24 us, 1,082 -> 739.
// The entries: the band's x faces, its y faces, its cells (DevState::mt).
__global__ void __launch_bounds__(256) k_maxwell_tab(DevState s, int faces) {
  pdl_wait();
  pdl_next();
  const Geo& g = s.g;
  const int nt = g.nu + g.nvel / g.nu, rows = s.mt_j1 - s.mt_j0;
  const int nfx = faces ? rows * (g.nx + 1) : 0, nf = faces ? nfx + (rows + 1) * g.nx : 0;
  const long t = (long)blockIdx.x * 256 + threadIdx.x;
  const int e = (int)(t / nt), a = (int)(t - (long)e * nt);
  if (e >= nf + g.nx * rows) return;
  const bool isu = a < g.nu;
  const double x = isu ? s.u[a] : s.v[(long)(a - g.nu) * g.nu];
  const double* tab = EXP64_TAB;
  const auto factor = [&](double amp, double U, double l2) {
    const double d = x - U, y = exp2_tab(l2, d * d, tab);
    return isu ? amp * y : y;  // the amplitude goes with the first axis
  };
  if (e < nf) {
    const int f = e < nfx ? s.mt_j0 * (g.nx + 1) + e : s.nface_x + s.mt_j0 * g.nx + (e - nfx);
    if (s.kind[f] == 0) return;
    const Quad64 E = s.fc64[f].E;
    // y faces: normal v, tangential -u
    const double U = e < nfx ? (isu ? E.y : E.z) : (isu ? -E.z : E.y);
    s.mt[(long)e * nt + a] = factor(E.x, U, E.w);
    return;
  }
  const int q = e - nf, j = q / g.nx;
  const CellParam& C = s.cp[cell_index(g, q - j * g.nx, s.mt_j0 + j)];
  if (!C.upd) return;
  const bool shak = s.coll == COLL_SHAKHOV;
  double* o = s.mt + ((long)nf + (shak ? 2L : 1L) * q) * nt + a;
  o[0] = factor(C.rho_n, isu ? C.U : C.V, C.l2);
  if (shak) o[nt] = factor(C.o_rho_n, isu ? C.oU : C.oV, EXP64_LOG2E * C.olam);
}

// residual = sqrt(sumRes N) / (sumAvg + 1e-7) + sqrt(boundary sumRes 2) / (...)
// (src/Solver/solver_update.jl:86-88, :239-241; update_boundary.jl:41-44, :284-288).
template <bool GRP = false>
__global__ void __launch_bounds__(256) k_residual(DevState sp) {
  pdl_wait();
  pdl_next();
  int lb;
  const int gr = group_member<GRP, GK_RES>(sp, lb);
  KB_GROUP_STATE(GRP, sp, gr);
  __shared__ double red[8][16];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double acc[16];
  for (int k = 0; k < 16; ++k) acc[k] = 0.0;
  for (int b = threadIdx.x; b < s.res_blocks; b += 256)
    for (int k = 0; k < 16; ++k) acc[k] += s.blockres[(long)b * 16 + k];
  const double sum = warp_sums<16>(acc, lane);
  if ((lane & 1) == 0) red[wid][lane >> 1] = sum;
  __syncthreads();
  if (wid != 0) return;
  double t = red[0][lane & 15];
  for (int k = 1; k < 8; ++k) t += red[k][lane & 15];
  // lane k < 4: component k (sums k and 4 + k of the interior, 8 + k and 12 + k
  // of the boundary cells)
  const double a = __shfl_down_sync(0xffffffffu, t, 4), b = __shfl_down_sync(0xffffffffu, t, 8),
               c = __shfl_down_sync(0xffffffffu, t, 12);
  if (lane < 4) {
    const Geo& g = s.g;
    double n = g.D == 1 ? double(g.nx) : double(g.nx) * g.ny;
    double r = sqrt(t * n) / (a + 1.e-7);
    r += sqrt(b * 2) / (c + 1.e-7);
    s.residual[lane] = r;
  }
}

// ------------------------------------------------------------ cell update

// Per-face constants of the update loop, built once per warp so the velocity
// loop runs in the storage precision only.
template <typename R>
struct FaceCtx {
  int kind;             // 0 none, 1 interior, 2 wall
  int cL, cR, step;     // cells on both sides and the cell step along the normal
  int ruleL, ruleR;     // slope rules of the two cells along the normal
  R dsc, dxh;           // 1/dx (FP32) or dx (FP64), dx/2
  FP<R> P;              // interior coefficients
  R wU, wV, wlam, wrn, wcB, wsc;  // wall: velocity, lambda, rho (lam/pi)^(D/2), K/(2 lam), len dt
  int rot;
};

template <typename R, int D>
__device__ __forceinline__ FaceCtx<R> make_ctx(const DevState& s, int f, int kind, bool right,
                                               double dt) {
  const Geo& g = s.g;
  FaceCtx<R> x;
  x.kind = kind;
  FaceGeo r = face_geo(g, f);
  x.cL = r.cL;
  x.cR = r.cR;
  x.step = r.step;
  x.ruleL = slope_rule(g, r.d, r.iL);
  x.ruleR = slope_rule(g, r.d, r.iR);
  double dd = r.d == 0 ? g.dx : g.dy;
  x.dsc = dscale<R>(dd);
  x.dxh = R(0.5 * dd);
  x.rot = right ? -1 : 1;
  if (kind == 1) x.P = load_fp<R>(s, f);
  if (kind == 2) {
    const double* wp = s.wall + (long)f * 4;
    double lw = D == 1 ? wp[2] : wp[3];
    double rho = s.rhow[f];
    x.wU = R(r.d == 0 ? wp[1] : wp[2]);
    x.wV = R(D == 1 ? 0.0 : (r.d == 0 ? wp[2] : -wp[1]));
    x.wlam = R(lw);
    x.wrn = R(D == 1 ? rho * sqrt64(lw * (1.0 / PI)) : rho * (lw * (1.0 / PI)));
    x.wcB = R(g.Kb * (0.5 * rcp64(lw)));
    x.wsc = R(D == 2 ? (r.d == 0 ? g.dy : g.dx) * dt : dt);
  }
  return x;
}

// Pointwise flux of one face at velocity v (face-local velocities un, ut);
// c is the interior cell next to a wall face.
template <typename R, int D, int FLUX>
__device__ __forceinline__ void ctx_flux(const FaceCtx<R>& x, const R* H,
                                         const R* Bq, long vs, int c, int v,
                                         R un, R ut, R dt, R& fh, R& fb) {
  if (x.kind == 0) {
    fh = R(0);
    fb = R(0);
    return;
  }
  if (x.kind == 2) {
    // u h_wall len dt with h_wall the wall Maxwellian on incoming velocities
    bool in = un * R(x.rot) >= R(0);
    R hw, bw;
    if (in) {
      R du = un - x.wU, e = du * du;
      if (D == 2) {
        R dv = ut - x.wV;
        e += dv * dv;
      }
      hw = x.wrn * mexp(-x.wlam * e);
      bw = hw * x.wcB;
    } else {
      hw = H[(long)c * vs + v];
      bw = Bq[(long)c * vs + v];
    }
    fh = un * hw * x.wsc;
    fb = un * bw * x.wsc;
    return;
  }
  bool pos = un >= R(0);
  int up = pos ? x.cL : x.cR;
  int rule = pos ? x.ruleL : x.ruleR;
  R sh, sb;
  R h = upwind_state<R>(H, vs, up, x.step, rule, pos, v, x.dsc, x.dxh, sh);
  R b = upwind_state<R>(Bq, vs, up, x.step, rule, pos, v, x.dsc, x.dxh, sb);
  R Th, Tb;
  face_flux<R, FLUX, D>(x.P, dt, un, ut, pos, h, b, sh, sb, fh, fb, Th, Tb);
}

// ------------------------------------------------------------ ghost fill

// copy_ctr! of w, prim, sw, h, b (src/Struct/struct.jl:55-66) for bc_extra!
// (src/Boundary/bc_extra.jl) and 1D bc_period! (src/Boundary/bc_period.jl:10-19)
// in the new buffers.  pass 0: x sides, pass 1: y sides.  One block per ghost cell.
template <typename R>
__global__ void k_ghost(DevState s, int pass) {
  pdl_wait();
  pdl_next();
  const Geo& g = s.g;
  int t = blockIdx.x;
  int dst = -1, src = -1;
  if (pass == 0) {
    int nrow = g.D == 2 ? g.nyt : 1;
    int per = 2 * g.ngx;
    if (t >= per * nrow) return;
    int jj = t / per, k = t % per;
    int j = jj - g.ngy;
    if (k < g.ngx) {  // left ghost 1-k-1 (0-based: -1-k)
      int gi = -1 - k;
      if (g.bc[0] == BC_EXTRA) src = cell_index(g, 0, j);
      else if (g.bc[0] == BC_PERIOD && g.D == 1) src = cell_index(g, g.nx - 1 - k, j);
      if (src >= 0) dst = cell_index(g, gi, j);
    } else {
      int kk = k - g.ngx;
      int gi = g.nx + kk;
      if (g.bc[1] == BC_EXTRA) src = cell_index(g, g.nx - 1, j);
      else if (g.bc[0] == BC_PERIOD && g.D == 1) src = cell_index(g, kk, j);
      if (src >= 0) dst = cell_index(g, gi, j);
    }
  } else {
    int per = 2 * g.ngy;
    if (t >= per * g.nxt) return;
    int ii = t / per, k = t % per;
    int i = ii - g.ngx;
    if (k < g.ngy) {
      if (g.bc[2] == BC_EXTRA) { src = cell_index(g, i, 0); dst = cell_index(g, i, -1 - k); }
    } else {
      int kk = k - g.ngy;
      if (g.bc[3] == BC_EXTRA) { src = cell_index(g, i, g.ny - 1); dst = cell_index(g, i, g.ny + kk); }
    }
  }
  if (dst < 0) return;
  R* Ho = (R*)s.h[s.cur ^ 1];
  R* Bo = (R*)s.b[s.cur ^ 1];
  long vs = g.vstride;
  for (int v = threadIdx.x; v < g.nvel; v += blockDim.x) {
    Ho[(long)dst * vs + v] = Ho[(long)src * vs + v];
    Bo[(long)dst * vs + v] = Bo[(long)src * vs + v];
  }
  if (threadIdx.x < 4) {
    s.w[(long)dst * 4 + threadIdx.x] = s.w[(long)src * 4 + threadIdx.x];
    s.prim[(long)dst * 4 + threadIdx.x] = s.prim[(long)src * 4 + threadIdx.x];
  }
  if (threadIdx.x < 8) s.sw[(long)dst * 8 + threadIdx.x] = s.sw[(long)src * 8 + threadIdx.x];
}

// ------------------------------------------------------------- dumps

template <typename R, int D, int FLUX>
__global__ void k_faces_dump(DevState s, double dt, double* fh_out, double* fb_out) {
  const Geo& g = s.g;
  int f = blockIdx.x;
  if (f >= s.nface_x + s.nface_y) return;
  int kind = s.kind[f];
  FaceGeo r = face_geo(g, f);
  const R* H = (const R*)s.h[s.cur];
  const R* Bq = (const R*)s.b[s.cur];
  const R* U = vtab<R>(s, 0);
  const R* V = vtab<R>(s, 1);
  int pos0 = r.d == 0 ? r.fi : r.fj;
  bool right = pos0 != 0;  // wall faces: the cell is on the left of the right / top wall
  int c = (kind == 2 && pos0 == 0) ? r.cR : r.cL;
  FaceCtx<R> X = make_ctx<R, D>(s, f, kind, right, dt);
  for (int v = threadIdx.x; v < g.nvel; v += blockDim.x) {
    R un, ut;
    if (D == 1) { un = U[v]; ut = R(0); }
    else if (r.d == 0) { un = U[v]; ut = V[v]; }
    else { un = V[v]; ut = -U[v]; }
    R fh = 0, fb = 0;
    ctx_flux<R, D, FLUX>(X, H, Bq, g.vstride, c, v, un, ut, R(dt), fh, fb);
    fh_out[(long)f * g.nvel + v] = double(fh);
    fb_out[(long)f * g.nvel + v] = double(fb);
  }
}

template <typename R>
__global__ void k_slopes_dump(DevState s, double* sh, double* sb) {
  const Geo& g = s.g;
  int c = blockIdx.x;
  int d = blockIdx.y;
  if (c >= s.ncell) return;
  int ci = c % g.nxt - g.ngx, cj = c / g.nxt - g.ngy;
  bool phys = ci >= 0 && ci < g.nx && cj >= 0 && cj < g.ny;
  int rule = phys ? slope_rule(g, d, d == 0 ? ci : cj) : 0;
  int step = d == 0 ? 1 : g.nxt;
  const R* H = (const R*)s.h[s.cur];
  const R* Bq = (const R*)s.b[s.cur];
  long vs = g.vstride;
  R dsc = dscale<R>(d == 0 ? g.dx : g.dy);
  for (int v = threadIdx.x; v < g.nvel; v += blockDim.x) {
    R t;
    R vh = upwind_state<R>(H, vs, c, step, rule, true, v, dsc, R(0), t);
    (void)vh;
    sh[((long)c * g.D + d) * g.nvel + v] = double(t);
    upwind_state<R>(Bq, vs, c, step, rule, true, v, dsc, R(0), t);
    sb[((long)c * g.D + d) * g.nvel + v] = double(t);
  }
}

// --------------------------------------------------------- conversions

// Row copy with conversion between the host layout ([cell][nvel], FP64) and
// the device layout ([cell][vstride], storage precision); a block converts cpb
// consecutive cells, threads striding over velocities (no index division).  Host
// arrays that are not 16-byte aligned take it.
template <typename DT, typename ST>
__global__ void k_conv(DT* __restrict__ dst, const ST* __restrict__ src, long ncell, int nvel,
                       int dvs, int svs, int cpb) {
  const long c0 = (long)blockIdx.x * cpb;
  for (int r = 0; r < cpb; ++r) {
    const long c = c0 + r;
    if (c >= ncell) return;
    for (int v = threadIdx.x; v < nvel; v += blockDim.x) dst[c * dvs + v] = (DT)src[c * svs + v];
  }
}
// The same conversion when both layouts are one dense array (nvel equal to
// the device row stride): element pairs, CONV_U of them per thread with all
// loads issued before the first store.  Across the host link (page-locked
// host arrays read or written in place) each load waits microseconds, so
// the bandwidth is the number of bytes in flight: 16-byte FP64 pairs, eight
// per thread.
constexpr int CONV_T = 256, CONV_U = 8;
template <typename T> struct ConvPair;
template <> struct ConvPair<float> {
  using T = float2;
  __device__ static float2 make(double a, double b) { return make_float2((float)a, (float)b); }
};
template <> struct ConvPair<double> {
  using T = double2;
  __device__ static double2 make(double a, double b) { return make_double2(a, b); }
};
template <typename DT, typename ST>
__global__ void __launch_bounds__(CONV_T) k_conv_flat(DT* __restrict__ dst, const ST* __restrict__ src,
                                                      long npair) {
  using S2 = typename ConvPair<ST>::T;
  using D2 = typename ConvPair<DT>::T;
  const long p0 = (long)blockIdx.x * (CONV_T * CONV_U) + threadIdx.x;
  S2 v[CONV_U];
#pragma unroll
  for (int u = 0; u < CONV_U; ++u) {
    const long p = p0 + (long)u * CONV_T;
    if (p < npair) v[u] = ((const S2*)src)[p];
  }
#pragma unroll
  for (int u = 0; u < CONV_U; ++u) {
    const long p = p0 + (long)u * CONV_T;
    if (p < npair) ((D2*)dst)[p] = ConvPair<DT>::make((double)v[u].x, (double)v[u].y);
  }
}
// Dense, even-length arrays whose pair loads and stores are aligned take the
// pair kernel.
static bool conv_flat_ok(const void* dst, size_t desz, const void* src, size_t sesz, int nvel, int vstride) {
  return nvel == vstride && nvel % 2 == 0 && (uintptr_t)dst % (2 * desz) == 0 &&
         (uintptr_t)src % (2 * sesz) == 0;
}
template <typename DT, typename ST>
static void conv_flat(DT* dst, const ST* src, long n, cudaStream_t st) {
  const long npair = n / 2;
  const unsigned nb = (unsigned)((npair + CONV_T * CONV_U - 1) / (CONV_T * CONV_U));
  k_conv_flat<DT, ST><<<nb, CONV_T, 0, st>>>(dst, src, npair);
}

// The conversion between dense host rows and padded device rows (OUT: to the
// host) by pairs of dense elements, so that the host side moves 16 aligned bytes
// a thread and whole lines a warp with all of a thread's loads in flight; rows
// of an odd number of elements, written row by row, cross the link in pieces.
// 12,707 cells x 1,073 velocities, h and b (226 MB): in 1,277 -> 1,204 us, out
// 1,505 -> 1,298 (174 GB/s).
template <typename T, bool OUT>
__global__ void __launch_bounds__(CONV_T) k_conv_rows(T* __restrict__ dev, double* __restrict__ host, long n,
                                                      unsigned nvel, int vs) {
  const long e0 = (long)blockIdx.x * (2 * CONV_T * CONV_U), c0 = e0 / nvel;
  const unsigned r0 = (unsigned)(e0 - c0 * nvel);
  T* base = dev + c0 * vs;
  double2 v[CONV_U];
  long o[CONV_U][2];
#pragma unroll
  for (int u = 0; u < CONV_U; ++u) {
    const unsigned off = 2 * (u * CONV_T + threadIdx.x), a = r0 + off, c = a / nvel, w = a - c * nvel;
    const long e = e0 + off;
    o[u][0] = (long)c * vs + w;
    o[u][1] = w + 1 == nvel ? (long)(c + 1) * vs : o[u][0] + 1;
    v[u] = make_double2(0.0, 0.0);
    if (OUT) {
      if (e < n) v[u].x = (double)base[o[u][0]];
      if (e + 1 < n) v[u].y = (double)base[o[u][1]];
    } else {
      if (e + 1 < n) v[u] = *(const double2*)(host + e);
      else if (e < n) v[u].x = host[e];
    }
  }
#pragma unroll
  for (int u = 0; u < CONV_U; ++u) {
    const long e = e0 + 2 * (u * CONV_T + (int)threadIdx.x);
    if (OUT) {
      if (e + 1 < n) *(double2*)(host + e) = v[u];
      else if (e < n) host[e] = v[u].x;
    } else {
      if (e < n) base[o[u][0]] = (T)v[u].x;
      if (e + 1 < n) base[o[u][1]] = (T)v[u].y;
    }
  }
}
template <typename T, bool OUT>
static void conv_rows(T* dev, double* host, long ncell, int nvel, int vs, cudaStream_t st) {
  const long n = ncell * nvel, per = 2L * CONV_T * CONV_U;
  k_conv_rows<T, OUT><<<(unsigned)((n + per - 1) / per), CONV_T, 0, st>>>(dev, host, n, (unsigned)nvel, vs);
}

// timestep: max over physical cells (src/Solver/solver_main.jl:240-342); one block.
// Maximum over the physical cells of the CFL rate; each block reduces its
// cells, then one atomic max per block on the bit pattern (the rates are
// positive, so their IEEE bits order like unsigned integers and the result
// does not depend on the order of the blocks).
__global__ void k_timestep(DevState s, double umax, double vmax, double* out) {
  __shared__ double red[256];
  const Geo& g = s.g;
  double m = 0.0;
  const long n = (long)g.nx * g.ny;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    int i = (int)(t % g.nx), j = (int)(t / g.nx);
    const double* p = s.prim + (long)cell_index(g, i, j) * 4;
    const double sos = sqrt64((0.5 * g.gamma) * rcp64(p[g.NW - 1]));
    double v = (fmax(umax, fabs(p[1])) + sos) * g.rdx;
    if (g.D == 2) v = fma(fmax(vmax, fabs(p[2])) + sos, g.rdy, v);
    m = fmax(m, v);
  }
  red[threadIdx.x] = m;
  __syncthreads();
  for (int st = 128; st >= 1; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + st]);
    __syncthreads();
  }
  if (threadIdx.x == 0)
    atomicMax((unsigned long long*)out, (unsigned long long)__double_as_longlong(red[0]));
}

// Equilibrium initial distributions of init_fvm (src/Solver/solver_init.jl:
// 119-141, :285-325): h = maxwellian(u, prim) (src/Theory/theory_equilibrium.jl:
// 8-25), b = h K / (2 lambda), for every cell incl. ghosts into buffer 0, and
// for ghost cells, which some boundaries never rewrite, into both buffers.
// One block per cell.
__device__ __forceinline__ bool ghost_cell(const Geo& g, long c) {
  const int i = (int)(c % g.nxt) - g.ngx, j = (int)(c / g.nxt) - g.ngy;
  return i < 0 || i >= g.nx || j < 0 || j >= g.ny;
}
constexpr int INIT_T = 128;
template <typename R>
__global__ void __launch_bounds__(INIT_T) k_init_eq(DevState s) {
  const Geo& g = s.g;
  const long c = blockIdx.x;
  const double* p = s.prim + c * 4;
  const double rho = p[0], U = p[1], V = g.D == 2 ? p[2] : 0.0, lam = p[g.NW - 1];
  const double rn = g.D == 1 ? rho * sqrt64(lam * (1.0 / PI)) : rho * (lam * (1.0 / PI));
  const double cB = g.Kb * (0.5 * rcp64(lam)), l2 = EXP64_LOG2E * lam;
  const int nb = ghost_cell(g, c) ? 2 : 1;
  for (int v = threadIdx.x; v < g.nvel; v += INIT_T) {
    const double du = s.u[v] - U;
    double e = du * du;
    if (g.D == 2) {
      const double dv = s.v[v] - V;
      e = fma(dv, dv, e);
    }
    const double M = rn * exp2_tab(l2, e, EXP64_TAB), MB = M * cB;
    for (int k = 0; k < nb; ++k) {
      ((R*)s.h[k])[c * g.vstride + v] = (R)M;
      ((R*)s.b[k])[c * g.vstride + v] = (R)MB;
    }
  }
}
// The same when the velocity grid is a product of nu and nv abscissae
// (Geo::tensor): the Maxwellian is then a product too, so a cell takes nu + nv
// exponentials instead of nu nv.  FP64: two products per point.  FP32: the
// factors and K / (2 lambda) as pairs of floats, whose products carry about 47
// bits before the one rounding to FP32, because the FP64 pipe would bound the
// kernel (512^2 cells x 64^2 velocities: 49.6 ms with an FP64 exponential per
// point, bound by writing h and b since).
struct F2 {
  float hi, lo;
};
__device__ __forceinline__ F2 f2_of(double x) {
  F2 r;
  r.hi = f32_of(x);
  r.lo = f32_of(x - f64_of(r.hi));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  r.hi = __fmul_rn(a.hi, b.hi);
  r.lo = fmaf(a.hi, b.hi, -r.hi) + fmaf(a.hi, b.lo, a.lo * b.hi);
  return r;
}
template <typename R> struct InitPart;
template <> struct InitPart<double> {
  using T = double;
  static __device__ double of(double x) { return x; }
  static __device__ double mul(double a, double b) { return a * b; }
  static __device__ double value(double a) { return a; }
};
template <> struct InitPart<float> {
  using T = F2;
  static __device__ F2 of(double x) { return f2_of(x); }
  static __device__ F2 mul(F2 a, F2 b) { return f2_mul(a, b); }
  static __device__ float value(F2 a) { return a.hi + a.lo; }
};
template <typename R>
__global__ void __launch_bounds__(INIT_T) k_init_eq_product(DevState s) {
  using IP = InitPart<R>;
  using T = typename IP::T;
  extern __shared__ __align__(16) unsigned char smi[];
  const Geo& g = s.g;
  const int nu = g.nu, nv = g.nvel / g.nu;
  T* su = (T*)smi;    // rho lambda / pi exp(-lambda (u - U)^2)
  T* sv = su + nu;    // exp(-lambda (v - V)^2)
  const long c = blockIdx.x;
  const double* p = s.prim + c * 4;
  const double U = p[1], V = p[2], lam = p[3], l2 = EXP64_LOG2E * lam, rn = p[0] * (lam * (1.0 / PI));
  const T cB = IP::of(g.Kb * (0.5 * rcp64(lam)));
  for (int k = threadIdx.x; k < nu + nv; k += INIT_T) {
    const bool first = k < nu;
    const double d = first ? s.u[k] - U : s.v[(k - nu) * nu] - V;
    const double e = exp2_tab(l2, d * d, EXP64_TAB);
    su[k] = IP::of(first ? rn * e : e);  // sv follows su
  }
  __syncthreads();
  const int nb = ghost_cell(g, c) ? 2 : 1;
  const int di = INIT_T % nu, dj = INIT_T / nu;
  int i = threadIdx.x % nu, j = threadIdx.x / nu;
  for (int v = threadIdx.x; v < g.nvel; v += INIT_T) {
    const T M = IP::mul(su[i], sv[j]);
    const R h = IP::value(M), b = IP::value(IP::mul(M, cB));
    for (int k = 0; k < nb; ++k) {
      ((R*)s.h[k])[c * g.vstride + v] = h;
      ((R*)s.b[k])[c * g.vstride + v] = b;
    }
    i += di;
    j += dj;
    if (i >= nu) {
      i -= nu;
      ++j;
    }
  }
}
// Ghost cells of buffer 0 into buffer 1 (after an upload); one block per ghost cell.
template <typename R>
__global__ void k_ghost_dup(DevState s) {
  const Geo& g = s.g;
  const int t = blockIdx.x, rows = 2 * g.ngy * g.nxt;
  int i, j;
  if (t < rows) {  // whole ghost rows
    const int r = t / g.nxt;
    i = t % g.nxt - g.ngx;
    j = r < g.ngy ? r - g.ngy : g.ny + r - g.ngy;
  } else {
    const int q = t - rows, k = q % (2 * g.ngx);
    j = q / (2 * g.ngx);
    i = k < g.ngx ? k - g.ngx : g.nx + k - g.ngx;
  }
  const long o = (long)cell_index(g, i, j) * g.vstride;
  for (int v = threadIdx.x; v < g.nvel; v += blockDim.x) {
    ((R*)s.h[1])[o + v] = ((R*)s.h[0])[o + v];
    ((R*)s.b[1])[o + v] = ((R*)s.b[0])[o + v];
  }
}

// ------------------------------------------------------------- launchers

// Launch of a step kernel in its chain (launch_after).
template <typename... P, typename... A>
static void go(void (*fn)(P...), unsigned blocks, int threads, cudaStream_t st, A... a) {
  std::tuple<P...> v(a...);
  std::apply([&](P&... x) {
    void* args[] = {(void*)&x...};
    launch_after((const void*)fn, dim3(blocks), dim3((unsigned)threads), 0, st, args);
  }, v);
}

static inline unsigned nblk(long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Every kernel of a step asks for the largest shared-memory carveout, the one
// the two HBM passes need for their rings.  An SM holds CTAs of kernels with
// different carveouts only after it drains and reconfigures, so when many
// solves share the GPU (a served stream: one CUDA stream per solve) a single
// carveout for all step kernels lets their CTAs share SMs.  Set once per
// kernel and device, on the first (uncaptured) launch.
void prefer_max_shared(const void* fn) {
  static std::mutex m;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(m);
  if (done.insert(std::make_pair(fn, dev)).second)
    cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                         cudaSharedmemCarveoutMaxShared);
}

// Threads per block of the one-thread-per-item FP64 kernels (w slopes, face
// parameters): one warp per block while the items fill fewer than two
// 128-thread blocks per multiprocessor, so a small grid spreads its FP64 work
// over more multiprocessors' FP64 pipes instead of queueing on a few.
static inline int item_bs(const DevState& s, long n) { return n < 2L * s.sm_count * 128 ? 32 : 128; }

int launch_reconstruct(DevState& s, cudaStream_t st) {
  if (s.flux == FLUX_KFVS) return 0;  // KFVS reads no w slopes
  long n = (long)s.g.nx * s.g.ny * s.g.D;
  if (s.g.interp == 1) return 0;
  const int bs = item_bs(s, n);
  prefer_max_shared((const void*)k_wslope<>);
  go(k_wslope<>, nblk(n, bs), bs, st, s);
  return 1;
}

template <int D>
static void (*face_param_fn(int flux, bool fast))(DevState, double) {
  switch (flux) {
    case FLUX_KFVS: return fast ? k_face_param<D, FLUX_KFVS, true> : k_face_param<D, FLUX_KFVS, false>;
    case FLUX_KCU: return fast ? k_face_param<D, FLUX_KCU, true> : k_face_param<D, FLUX_KCU, false>;
    default: return fast ? k_face_param<D, FLUX_UGKS, true> : k_face_param<D, FLUX_UGKS, false>;
  }
}

int launch_face_param(DevState& s, double dt, cudaStream_t st) {
  int nf = s.nface_x + s.nface_y;
  const bool fast = s.prec != 0;
  const int bs = item_bs(s, nf);
  void (*fn)(DevState, double) = s.g.D == 2 ? face_param_fn<2>(s.flux, fast) : face_param_fn<1>(s.flux, fast);
  prefer_max_shared((const void*)fn);
  go(fn, nblk(nf, bs), bs, st, s, dt);
  return 1;
}

// The factors of the step's Maxwellians (DevState::mt) of the band's faces, when
// the flux evaluates them, and of its cells.
int launch_maxwell_tab(const DevState& s, bool faces, cudaStream_t st) {
  const long rows = s.mt_j1 - s.mt_j0, nx = s.g.nx;
  const long n = ((faces ? (nx + 1) * rows + nx * (rows + 1) : 0) + nx * rows) * (s.g.nu + s.g.nvel / s.g.nu);
  prefer_max_shared((const void*)k_maxwell_tab);
  go(k_maxwell_tab, (unsigned)((n + 255) / 256), 256, st, s, faces ? 1 : 0);
  return 1;
}

int launch_wall(DevState& s, double dt, cudaStream_t st) {
  if (s.nwall == 0) return 0;
  void (*fn)(DevState, double);
  if (s.g.D == 1) fn = s.prec == 0 ? k_wall<double, 1> : k_wall<float, 1>;
  else fn = s.prec == 0 ? k_wall<double, 2> : k_wall<float, 2>;
  prefer_max_shared((const void*)fn);
  go(fn, (unsigned)s.nwall, WALL_T, st, s, dt);
  return 1;
}

int launch_evolve(DevState& s, double dt, cudaStream_t st) {
  int n = launch_face_param(s, dt, st);
  n += launch_moments(s, dt, true, st);
  return n;
}

template <int BS>
static void cell_param_bs(DevState& s, double dt, bool res, cudaStream_t st) {
  const bool fast = s.prec != 0;
  void (*fn)(DevState, double, int);
  if (s.g.D == 1) fn = fast ? k_cell_param<1, true, BS> : k_cell_param<1, false, BS>;
  else fn = fast ? k_cell_param<2, true, BS> : k_cell_param<2, false, BS>;
  prefer_max_shared((const void*)fn);
  go(fn, (unsigned)s.res_blocks, BS, st, s, dt, res ? 1 : 0);
}

int launch_cell_param(DevState& s, double dt, cudaStream_t st, bool res) {
  if (s.cell_bs == 32) cell_param_bs<32>(s, dt, res, st);
  else cell_param_bs<256>(s, dt, res, st);
  return 1;
}

template <typename R, int D>
static int finish_t(DevState& s, cudaStream_t st, bool res) {
  int n = 0;
  s.cur ^= 1;
  bool fill = false;
  for (int k = 0; k < 2 * D; ++k) fill |= s.g.bc[k] == BC_EXTRA || s.g.bc[k] == BC_PERIOD;
  if (fill) {
    // the ghost kernels write into buffer cur^1 of their DevState copy: pass
    // a copy that still points at the pre-swap index so they fill the new state
    DevState t = s;
    t.cur ^= 1;
    int nrow = D == 2 ? s.g.nyt : 1;
    prefer_max_shared((const void*)k_ghost<R>);
    if (s.g.ngx > 0) { go(k_ghost<R>, (unsigned)(2 * s.g.ngx * nrow), 128, st, t, 0); ++n; }
    if (D == 2 && s.g.ngy > 0) { go(k_ghost<R>, (unsigned)(2 * s.g.ngy * s.g.nxt), 128, st, t, 1); ++n; }
  }
  if (res) {
    prefer_max_shared((const void*)k_residual<false>);
    go(k_residual<false>, 1u, 256, st, s);
    ++n;
  }
  return n;
}

// ---- grouped launches (kb_group.cu): the per-face / per-cell kernels of one
// step of the 2D FP32 form over all members of a group; ls.grp points at
// the step's member table, the block counts are the members' summed.
void group_small(int kind, const DevState& ls, int flux, int blocks, bool res, cudaStream_t st) {
  if (blocks <= 0) return;
  const void* fn = nullptr;
  switch (kind) {
    case GK_WSLOPE:
      fn = (const void*)k_wslope<true>;
      prefer_max_shared(fn);
      go(k_wslope<true>, (unsigned)blocks, 32, st, ls);
      break;
    case GK_FACE: {
      void (*f)(DevState, double) = flux == FLUX_KFVS ? k_face_param<2, FLUX_KFVS, true, true>
                                    : flux == FLUX_KCU ? k_face_param<2, FLUX_KCU, true, true>
                                                       : k_face_param<2, FLUX_UGKS, true, true>;
      prefer_max_shared((const void*)f);
      go(f, (unsigned)blocks, 32, st, ls, 0.0);
      break;
    }
    case GK_CELL:
      fn = (const void*)k_cell_param<2, true, 32, true>;
      prefer_max_shared(fn);
      go(k_cell_param<2, true, 32, true>, (unsigned)blocks, 32, st, ls, 0.0, res ? 1 : 0);
      break;
    case GK_RES:
      fn = (const void*)k_residual<true>;
      prefer_max_shared(fn);
      go(k_residual<true>, (unsigned)blocks, 256, st, ls);
      break;
    default:
      break;
  }
}

int launch_finish(DevState& s, cudaStream_t st, bool res) {
  if (s.prec == 0) return s.g.D == 1 ? finish_t<double, 1>(s, st, res) : finish_t<double, 2>(s, st, res);
  return s.g.D == 1 ? finish_t<float, 1>(s, st, res) : finish_t<float, 2>(s, st, res);
}

int launch_update(DevState& s, double dt, cudaStream_t st, bool res) {
  int n = launch_cell_param(s, dt, st, res);
  n += launch_march(s, dt, st);
  n += launch_finish(s, st, res);
  return n;
}

template <typename R, int D>
static int faces_dump_t(DevState& s, double dt, double* fh, double* fb, cudaStream_t st) {
  int nf = s.nface_x + s.nface_y;
  switch (s.flux) {
    case FLUX_KFVS: k_faces_dump<R, D, FLUX_KFVS><<<nf, 128, 0, st>>>(s, dt, fh, fb); break;
    case FLUX_KCU: k_faces_dump<R, D, FLUX_KCU><<<nf, 128, 0, st>>>(s, dt, fh, fb); break;
    default: k_faces_dump<R, D, FLUX_UGKS><<<nf, 128, 0, st>>>(s, dt, fh, fb); break;
  }
  return 1;
}

int launch_faces_dump(DevState& s, double dt, double* fh, double* fb, cudaStream_t st) {
  if (s.prec == 0)
    return s.g.D == 1 ? faces_dump_t<double, 1>(s, dt, fh, fb, st) : faces_dump_t<double, 2>(s, dt, fh, fb, st);
  return s.g.D == 1 ? faces_dump_t<float, 1>(s, dt, fh, fb, st) : faces_dump_t<float, 2>(s, dt, fh, fb, st);
}

int launch_slopes_dump(DevState& s, double* sh, double* sb, cudaStream_t st) {
  dim3 grid(s.ncell, s.g.D);
  if (s.prec == 0) k_slopes_dump<double><<<grid, 128, 0, st>>>(s, sh, sb);
  else k_slopes_dump<float><<<grid, 128, 0, st>>>(s, sh, sb);
  return 1;
}

int launch_convert_in(void* dst, int prec, const double* src, long ncell, int nvel, int vstride,
                      cudaStream_t st) {
  if (ncell * nvel == 0) return 0;
  if (conv_flat_ok(dst, prec == 0 ? 8 : 4, src, 8, nvel, vstride)) {
    if (prec == 0) conv_flat((double*)dst, src, ncell * nvel, st);
    else conv_flat((float*)dst, src, ncell * nvel, st);
    return 1;
  }
  if ((uintptr_t)src % 16 == 0) {
    if (prec == 0) conv_rows<double, false>((double*)dst, (double*)src, ncell, nvel, vstride, st);
    else conv_rows<float, false>((float*)dst, (double*)src, ncell, nvel, vstride, st);
    return 1;
  }
  const int cpb = std::max(1, 2048 / nvel);
  const unsigned nb = (unsigned)((ncell + cpb - 1) / cpb);
  if (prec == 0) k_conv<double, double><<<nb, 256, 0, st>>>((double*)dst, src, ncell, nvel, vstride, nvel, cpb);
  else k_conv<float, double><<<nb, 256, 0, st>>>((float*)dst, src, ncell, nvel, vstride, nvel, cpb);
  return 1;
}

int launch_convert_out(double* dst, int prec, const void* src, long ncell, int nvel, int vstride,
                       cudaStream_t st) {
  if (ncell * nvel == 0) return 0;
  if (conv_flat_ok(dst, 8, src, prec == 0 ? 8 : 4, nvel, vstride)) {
    if (prec == 0) conv_flat(dst, (const double*)src, ncell * nvel, st);
    else conv_flat(dst, (const float*)src, ncell * nvel, st);
    return 1;
  }
  if ((uintptr_t)dst % 16 == 0) {
    if (prec == 0) conv_rows<double, true>((double*)src, dst, ncell, nvel, vstride, st);
    else conv_rows<float, true>((float*)src, dst, ncell, nvel, vstride, st);
    return 1;
  }
  const int cpb = std::max(1, 2048 / nvel);
  const unsigned nb = (unsigned)((ncell + cpb - 1) / cpb);
  if (prec == 0)
    k_conv<double, double><<<nb, 256, 0, st>>>(dst, (const double*)src, ncell, nvel, nvel, vstride, cpb);
  else
    k_conv<double, float><<<nb, 256, 0, st>>>(dst, (const float*)src, ncell, nvel, nvel, vstride, cpb);
  return 1;
}

int launch_timestep(const DevState& s, double umax, double vmax, double* out, cudaStream_t st) {
  cudaMemsetAsync(out, 0, sizeof(double), st);
  const long n = (long)s.g.nx * s.g.ny;
  const unsigned nb = (unsigned)std::min<long>(1184, std::max<long>(1, (n + 255) / 256));
  k_timestep<<<nb, 256, 0, st>>>(s, umax, vmax, out);
  return 1;
}

int launch_init_equilibrium(DevState& s, cudaStream_t st) {
  const Geo& g = s.g;
  const size_t smem = 8 * (size_t)(g.nu + g.nvel / g.nu);
  if (g.tensor && smem <= 48 * 1024) {
    if (s.prec == 0) k_init_eq_product<double><<<s.ncell, INIT_T, smem, st>>>(s);
    else k_init_eq_product<float><<<s.ncell, INIT_T, smem, st>>>(s);
  } else if (s.prec == 0) {
    k_init_eq<double><<<s.ncell, INIT_T, 0, st>>>(s);
  } else {
    k_init_eq<float><<<s.ncell, INIT_T, 0, st>>>(s);
  }
  return 1;
}

int launch_ghost_dup(DevState& s, cudaStream_t st) {
  const int n = s.ncell - s.g.nx * s.g.ny;
  if (n == 0) return 0;
  if (s.prec == 0) k_ghost_dup<double><<<n, 128, 0, st>>>(s);
  else k_ghost_dup<float><<<n, 128, 0, st>>>(s);
  return 1;
}

}  // namespace kb
