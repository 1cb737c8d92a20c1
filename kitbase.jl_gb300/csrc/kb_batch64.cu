// kb_batch64.cu -- FP64 step of 1D2F1V solves (KFVS, fixed ends, van Leer),
// one CTA per segment of a few cells, the whole step fused in one launch.
#include "kb_batch64.cuh"

#include <algorithm>

#include "kb_f64.cuh"

namespace kb {

constexpr int SEG64_T = 256;  // against 128: 700 x 200 points 34.1 -> 28.3 us a step
constexpr int SEG64_CC = 12;  // doubles of coefficients per cell

int seg64_smem(int seg, int ns) {
  return 8 * ((2 * (seg + 4) + 2 * (seg + 1) + 5) * ns + (seg + 1) * 4 + seg * (SEG64_CC + 4) + EXP64_N + 8);
}

// The FP64 pipe bounds the step, and one warp on each quarter of a
// multiprocessor nearly fills it: the segments should give every
// multiprocessor the same work.  A segment of s cells forms s + 1 faces and
// has a fixed part worth about one more, so the length with the smallest
// (segments of the busiest multiprocessor) (s + 2) is taken.  Against four or
// more short segments per multiprocessor: 700 x 64 points 25.1 -> 13.8 us a
// step, 700 x 200 46.1 -> 28.3, 2048 x 256 106.8 -> 91.5; up to 16 cells a
// segment, whose memory leaves one CTA on a multiprocessor, are slower for
// ensembles (128 shocks: 753 against 650 us).
int seg64_cells(long cells, int sms) {
  long best = 0;
  int seg = 1;
  for (int s = 1; s <= SEG64_MAX; ++s) {
    const long ctas = (cells + s - 1) / s, t = (ctas + sms - 1) / std::max(1, sms) * (s + 2);
    if (s == 1 || t <= best) {
      best = t;
      seg = s;
    }
  }
  return seg;
}

// Sum of four values over the warp: a reduce-scatter (two exchanges that
// halve the number of values a lane carries, then three plain levels), 6
// FP64 additions instead of 20.  Lanes 0 .. 7 return the total of a, 8 .. 15 of
// b, 16 .. 23 of c, 24 .. 31 of d.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d, int lane) {
  const unsigned all = 0xffffffffu;
  const bool hi = lane & 16, mid = lane & 8;
  // level 16: the lower half keeps (a, b), the upper half (c, d)
  double k0 = hi ? c : a, k1 = hi ? d : b;
  const double g0 = hi ? a : c, g1 = hi ? b : d;
  k0 += __shfl_xor_sync(all, g0, 16);
  k1 += __shfl_xor_sync(all, g1, 16);
  // level 8: bit 8 clear keeps the first of the two, set the second
  double k = mid ? k1 : k0;
  const double g = mid ? k0 : k1;
  k += __shfl_xor_sync(all, g, 8);
  k += __shfl_xor_sync(all, k, 4);
  k += __shfl_xor_sync(all, k, 2);
  k += __shfl_xor_sync(all, k, 1);
  return k;
}

// Coefficients of a cell's Maxwellian from its prim [rho, U, lambda]: density
// factor, K / (2 lambda), and the Shakhov factor 0.8 (1 - Pr) lambda^2 / rho.
// A step needs them for the new state and for the old; the old ones are those
// that the step before formed from the same prim (BatchDev::mc64).
__device__ __forceinline__ void seg_coef64(const BatchDev& B, const double* p, double rrho, double* m) {
  m[0] = p[0] * sqrt64(p[2] * (1.0 / PI));
  m[1] = (0.5 * B.K) * rcp64(p[2]);
  m[2] = (0.8 * (1.0 - B.Pr)) * (p[2] * p[2]) * rrho;
}

// Segment k covers cells [seg_i0[k], seg_i0[k] + seg) of instance seg_b[k];
// its window (two more cells on each side, h and b, all velocities) arrives
// by two bulk copies.  Phases, a CTA barrier between them:
//   1  flux of every face of the segment at every velocity into shared memory
//      (each is used twice below: by its moments and by the two cells)
//   2  a warp per face: the three moments, and with them the old heat flux of
//      the cell to the right of the face
//   3  a lane per cell: w, prim, tau and the coefficients of the relaxation
//   4  relaxation of every (cell, velocity)
// Bound by the FP64 pipe: about 50 (BGK) or 80 (Shakhov) FP64 instructions per
// cell and velocity.  One CTA per instance, which formed every face flux twice
// with two IEEE divisions each, left 24 instances (7.5e5 cell-velocity points)
// on 24 multiprocessors: 4.24 ms a step, now 0.15 ms.  Results do not depend on the
// segment length or on what else is in the launch: a face's moments are
// summed in the same lane order wherever the segment starts.
__global__ void __launch_bounds__(SEG64_T) k_batch_seg64(BatchDev B, int seg, int nsm,
                                                         const double* Hin,
                                                         const double* Bin,
                                                         double* __restrict__ Hout,
                                                         double* __restrict__ Bout, int want_res,
                                                         int slot) {
  extern __shared__ __align__(16) unsigned char sm64[];
  __shared__ unsigned long long bar;
  __shared__ double sdt;     // dt
  __shared__ int sflag[2];   // the step is skipped; its residual and face moments are kept
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int k = blockIdx.x;
  const int b = B.seg_b[k], i0 = B.seg_i0[k];
  const int nx = B.nx[b], ng = B.ng[b], nu = B.nu[b], ns = B.nus[b];
  const int i1 = min(i0 + seg, nx);
  const long c0 = B.cell_off[b], e0 = B.elem_off[b];
  const double* Hi = Hin + e0;
  const double* Bi = Bin + e0;
  double* Ho = Hout + e0;
  double* Bo = Bout + e0;
  double* sH = (double*)sm64;
  double* sB = sH + (seg + 4) * nsm;
  double* sF = sB + (seg + 4) * nsm;  // fh [face][v]
  double* sG = sF + (seg + 1) * nsm;  // fb
  double* sU = sG + (seg + 1) * nsm;
  double* sW = sU + nsm;
  double* sWu = sW + nsm;             // weight * u
  double* sT = sWu + nsm;             // dt u
  double* sK = sT + nsm;              // +-dt u / 2 - dt^2 u^2 / (2 dx): factor of the slope
  double* sfw = sK + nsm;             // [face][4]
  double* sq = sfw + (seg + 1) * 4;   // [cell][4] old heat flux (first value)
  double* scc = sq + seg * 4;         // [cell][SEG64_CC]
  double* stab = scc + seg * SEG64_CC;  // 2^(j / 256)
  for (int v = tid; v < nu; v += SEG64_T) {
    const double u = B.u[B.vel_off[b] + v], w = B.wt[B.vel_off[b] + v];
    sU[v] = u;
    sW[v] = w;
    sWu[v] = w * u;
  }
  exp64_load(stab, tid, SEG64_T);
  // up to here only what no step writes
  pdl_wait();
  pdl_next();
  if (tid == 0) {
    SegClock c = {B.dt[b], 0.0, B.active[b] == 0, false};
    if (slot >= 0) {
      c = seg_clock(B, slot);
      if (k == 0) seg_clock_next(B, slot, c);
    }
    sdt = c.dt;
    sflag[0] = c.stop;
    sflag[1] = want_res || c.last;
    mbar_init(&bar, 1);
    fence_async_smem();
  }
  __syncthreads();
  if (sflag[0]) {  // converged or past the end: carry this segment's cells over
    for (long t = tid; t < (long)(i1 - i0) * ns; t += SEG64_T) {
      const long o = (long)(i0 + ng) * ns + t;
      Ho[o] = Hi[o];
      Bo[o] = Bi[o];
    }
    return;
  }
  // window rows r0 .. r1-1 (cells incl. ghosts) are contiguous in h and b
  const int r0 = max(i0 - 2, -ng), r1 = min(i1 + 2, nx + ng), nrow = r1 - r0;
  if (tid == 0) {
    const unsigned bytes = (unsigned)nrow * ns * 8u;
    mbar_expect(&bar, 2u * bytes);
    bulk_g2s(sH, Hi + (long)(r0 + ng) * ns, bytes, &bar);
    bulk_g2s(sB, Bi + (long)(r0 + ng) * ns, bytes, &bar);
  }
  const double dx = B.dx[b], dt = sdt;
  const double rdx = B.rdx[b];
  const double T4 = 0.5 * dt * dt * rdx;
  const int ca = max(i0, 1), cb = min(i1, nx - 1);  // stepped cells [ca, cb)
  const int nc = max(0, cb - ca), nf = nc > 0 ? nc + 1 : 0;  // faces ca .. cb
  const bool want = sflag[1] != 0;
  // the lane that updates a cell (of a warp that changes from segment to
  // segment: its number decides which quarter of the multiprocessor works)
  // reads its w and prim while the window is on its way
  const bool shak = B.coll == COLL_SHAKHOV;
  const int role = (wid + (int)(((unsigned)k * 2654435761u) >> 30)) % (SEG64_T / 32);
  const bool mine = role == 0 && lane < nc;
  const long cell = c0 + ca + lane + ng;
  double wo[3] = {1.0, 0.0, 1.0}, po[3] = {1.0, 0.0, 1.0}, mo[3] = {1.0, 0.0, 0.0}, rmu = 1.0;
  if (mine) {
    for (int m = 0; m < 3; ++m) {
      wo[m] = B.w[cell * 4 + m];
      po[m] = B.prim[cell * 4 + m];
      mo[m] = B.mc64[cell * 4 + m];
    }
    rmu = B.rmu[b];
  }
  for (int v = tid; v < nu; v += SEG64_T) {
    const double u = sU[v];
    const double tu = dt * u;
    sT[v] = tu;
    sK[v] = fma(nonneg64(u) ? 0.5 : -0.5, tu, -T4 * (u * u));
  }
  if (mine && shak) {  // the old Maxwellian
    double* cc = scc + lane * SEG64_CC;
    cc[7] = po[1];
    cc[8] = EXP64_LOG2E * po[2];
    cc[9] = mo[1];
    cc[10] = mo[0] * mo[2];
    cc[11] = 2.0 * po[2];
  }
  const bool ok = tid == 0 ? mbar_wait(&bar, 0) : true;
  if (__syncthreads_or(!ok)) {  // CTA-uniform: bounded clean-up, then leave
    if (tid == 0) {
      atomicOr(B.status, 2);
      if (slot >= 0) seg_clock_max(B, slot, seg_no_rate());
      mbar_wait(&bar, 0);
    }
    return;
  }
  const double epsd = 1.e-7 * dx;
  // ---- 1: fluxes.  fh = dt u (h + side s) - dt^2 u^2 / (2 dx) s = T h + K s
  const auto flux = [&](int f, int v, double& fh, double& fb) {
    const int up = f - (nonneg64(sU[v]) ? 1 : 0);  // upwind cell
    const int o = (up - r0) * ns + v;
    const double h0 = sH[o], b0 = sB[o];
    double sh = 0.0, sb = 0.0;
    if (brule(up, nx, ng) == 1) {
      sh = vl64(sH[o - ns], h0, sH[o + ns], epsd);
      sb = vl64(sB[o - ns], b0, sB[o + ns], epsd);
    }
    fh = fma(sK[v], sh, sT[v] * h0);
    fb = fma(sK[v], sb, sT[v] * b0);
  };
  for (int t = tid; t < nf * nu; t += SEG64_T) {
    const int j = t / nu, v = t - j * nu;
    flux(ca + j, v, sF[j * ns + v], sG[j * ns + v]);
  }
  __syncthreads();
  // ---- 2: moments of face ca + j and heat flux of cell ca + j
  for (int j = wid; j < nf; j += SEG64_T / 32) {
    double m0 = 0.0, m1 = 0.0, m2 = 0.0, q = 0.0;
    const double* F = sF + j * ns;
    const double* G = sG + j * ns;
    for (int v = lane; v < nu; v += 32) {
      const double fh = F[v], w = sW[v], wu = sWu[v];
      m0 = fma(w, fh, m0);
      m1 = fma(wu, fh, m1);
      m2 = fma(wu * sU[v], fh, fma(w, G[v], m2));
    }
    if (shak && j < nc) {
      const int o = (ca + j - r0) * ns;
      const double Uc = scc[j * SEG64_CC + 7];
      for (int v = lane; v < nu; v += 32) {
        const double cu = sU[v] - Uc;
        q = fma(sW[v] * cu, fma(cu * cu, sH[o + v], sB[o + v]), q);
      }
    }
    const double s = warp_sum4(m0, m1, m2, q, lane);
    if ((lane & 7) == 0) {
      const int m = lane >> 3;
      if (m < 3) sfw[j * 4 + m] = m == 2 ? 0.5 * s : s;
      else if (j < nc) sq[j * 4] = 0.5 * s;
    }
  }
  __syncthreads();
  // ---- 3: cell parameters, one lane per cell
  if (role == 0) {
    double rr[6] = {0, 0, 0, 0, 0, 0};
    double rate = 0.0;
    if (mine) {
      double* w = B.w + cell * 4;
      double* p = B.prim + cell * 4;
      const double* fL = sfw + lane * 4;
      const double* fR = fL + 4;
      double wn[3], pn[3];
      for (int m = 0; m < 3; ++m) wn[m] = wo[m] + (fL[m] - fR[m]) * rdx;
      // conserve_prim (src/Theory/theory_macro.jl:185-206) with hg = 0.5 / (gamma - 1)
      const double rr0 = rcp64(wn[0]), hr = wn[0] * B.hg;
      pn[0] = wn[0];
      pn[1] = wn[1] * rr0;
      const double ei = fma(-0.5 * wn[1], pn[1], wn[2]);
      const double lam = hr * rcp64(ei);
      pn[2] = lam;
      // dt / tau, tau = 2 mu lambda^(1 - omega) / rho (vhs_collision_time,
      // src/Theory/theory_relaxation.jl:28)
      const double dtau = (dt * rmu) * (pn[0] * pow_tab(lam, B.tau_pow, stab));
      double mn[3];
      seg_coef64(B, pn, rr0, mn);
      double* cc = scc + lane * SEG64_CC;
      cc[0] = mn[0];  // new Maxwellian
      cc[1] = pn[1];
      cc[2] = EXP64_LOG2E * lam;
      cc[3] = mn[1];
      cc[4] = dtau;
      cc[5] = rcp64(1.0 + dtau);
      if (shak) cc[10] *= sq[lane * 4];  // the factor of the heat flux
      for (int m = 0; m < 3; ++m) {
        w[m] = wn[m];
        p[m] = pn[m];
        B.mc64[cell * 4 + m] = mn[m];
      }
      if (want) {
        for (int m = 0; m < 3; ++m) {
          const double d = wn[m] - wo[m];
          rr[m] = d * d;
          rr[3 + m] = fabs(wn[m]);
        }
      }
      const bool good = pos64(pn[0]) && pos64(lam);
      if (!good) atomicOr(B.status, 1);
      if (slot >= 0) rate = good ? seg_rate(B, pn, rdx) : seg_no_rate();
    }
    if (want) {
#pragma unroll
      for (int m = 0; m < 6; ++m) rr[m] = warp_sum(rr[m]);
      if (lane == 0) {
        double* pr = B.respart + (long)k * 8;
#pragma unroll
        for (int m = 0; m < 6; ++m) pr[m] = rr[m];
      }
    }
    if (slot >= 0) seg_clock_rate(B, slot, rate, c0, ng, i0, i1, nx, rdx, lane);
  }
  __syncthreads();
  // ---- 4: relaxation; fixed end cells keep their state
  for (int v = tid; v < nu; v += SEG64_T) {
    if (i0 == 0) {
      Ho[(long)ng * ns + v] = sH[(0 - r0) * ns + v];
      Bo[(long)ng * ns + v] = sB[(0 - r0) * ns + v];
    }
    if (i1 == nx) {
      Ho[(long)(nx - 1 + ng) * ns + v] = sH[(nx - 1 - r0) * ns + v];
      Bo[(long)(nx - 1 + ng) * ns + v] = sB[(nx - 1 - r0) * ns + v];
    }
  }
  const double K3 = B.K - 3.0;
  for (int t = tid; t < nc * nu; t += SEG64_T) {
    const int j = t / nu, v = t - j * nu;
    const double* cc = scc + j * SEG64_CC;
    const int o = (ca + j - r0) * ns + v;
    const double u = sU[v];
    const double du = u - cc[1];
    double MH = cc[0] * exp2_tab(cc[2], du * du, stab);
    double MB = MH * cc[3];
    if (shak) {
      const double ou = u - cc[7], o2 = ou * ou;
      const double S = cc[10] * ou * exp2_tab(cc[8], o2, stab);
      const double tl = fma(cc[11], o2, K3);  // 2 lambda c^2 + K - 3
      MH = fma(S, tl - 2.0, MH);
      MB = fma(S * tl, cc[9], MB);
    }
    const long g = (long)(ca + j + ng) * ns + v;
    const double* F = sF + j * ns + v;
    const double* G = sG + j * ns + v;
    Ho[g] = fma(cc[4], MH, fma(F[0] - F[ns], rdx, sH[o])) * cc[5];
    Bo[g] = fma(cc[4], MB, fma(G[0] - G[ns], rdx, sB[o])) * cc[5];
  }
  // BatchDev::fw: the segment's faces but its first (the segment's before, if that
  // steps any), and with ghosts those of the ends, which no cell reads
  if (want && B.fw) {
    for (int t = tid; t < nf * 3; t += SEG64_T) {
      const int j = t / 3, m = t - j * 3;
      if (ca + j > i0 || ca + j == 1) B.fw[(long)(ca + j) * 4 + m] = sfw[j * 4 + m];
    }
    const bool end = wid == 1 ? i0 == 0 : (wid == 2 && i1 == nx);
    if (end && ng > 0) {
      const int f = wid == 1 ? 0 : nx;
      double m0 = 0.0, m1 = 0.0, m2 = 0.0;
      for (int v = lane; v < nu; v += 32) {
        double fh, fb;
        flux(f, v, fh, fb);
        m0 = fma(sW[v], fh, m0);
        m1 = fma(sWu[v], fh, m1);
        m2 = fma(sWu[v] * sU[v], fh, fma(sW[v], fb, m2));
      }
      const double s = warp_sum4(m0, m1, m2, 0.0, lane);
      const int m = lane >> 3;
      if ((lane & 7) == 0 && m < 3) B.fw[(long)f * 4 + m] = m == 2 ? 0.5 * s : s;
    }
  }
}

__global__ void k_batch_mcache64(BatchDev B) {
  const int b = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= B.nx[b] + 2 * B.ng[b]) return;
  const long cell = B.cell_off[b] + c;
  double mn[3];
  seg_coef64(B, B.prim + cell * 4, rcp64(B.prim[cell * 4]), mn);
  for (int m = 0; m < 3; ++m) B.mc64[cell * 4 + m] = mn[m];
}
void seg64_mcache_launch(const BatchDev& B, int n, int max_cells, cudaStream_t st) {
  k_batch_mcache64<<<dim3((unsigned)((max_cells + 31) / 32), (unsigned)n), 32, 0, st>>>(B);
}

bool seg64_prepare() {
  const bool ok = cudaFuncSetAttribute(k_batch_seg64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       seg64_smem(SEG64_MAX, SEG_MAXNU)) == cudaSuccess;
  prefer_max_shared((const void*)k_batch_seg64);
  return ok;
}

cudaError_t seg64_launch(const BatchDev& B, int seg, const double* hin, const double* bin, double* hout,
                         double* bout, bool want_res, int slot, cudaStream_t st) {
  if (B.nseg_all <= 0) return cudaSuccess;
  int nsm = B.nu4_max, res = want_res ? 1 : 0;
  void* args[] = {(void*)&B, &seg, &nsm, &hin, &bin, &hout, &bout, &res, &slot};
  return launch_after((const void*)k_batch_seg64, dim3((unsigned)B.nseg_all), dim3(SEG64_T),
                      (size_t)seg64_smem(seg, B.nu4_max), st, args);
}

}  // namespace kb
