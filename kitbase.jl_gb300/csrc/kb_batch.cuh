// kb_batch.cuh -- device side of the batched 1D2F1V solves: the ragged
// layout (BatchDev) and the fused FP32 segment kernel, a template over the
// segment length and the CTA size so that the autotuner can choose them
// (instantiated in kb_batch_seg_a.cu / kb_batch_seg_b.cu).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>
#include <vector>

#include "kb_device.cuh"
#include "kb_f64.cuh"
#include "kb_kernels.cuh"
#include "kb_tma.cuh"

namespace kb {

// What a segment CTA needs before it can ask for its window, in one load.
struct alignas(16) SegDesc {
  int b, i0;              // instance, first cell
  int nx, ng, nu, ns;     // the instance's (BatchDev)
  int vo, pad;            // velocity table offset
  long c0, e0;            // first cell, first distribution element
  double rdx;             // 1 / dx
  float epsd, mu2;        // 1e-7 dx, 2 mu
};
static_assert(sizeof(SegDesc) == 64, "four 16-byte loads");

struct BatchDev {
  int n;                 // instances
  const int* nx;         // physical cells
  const int* ng;         // ghost layers
  const int* nu;         // velocities
  const int* nus;        // row stride of the distributions: nu rounded up to 4
  const long* cell_off;  // first cell (incl. ghosts)
  const long* elem_off;  // first distribution element
  const int* vel_off;    // velocity table offset
  const double* dx;      // cell size
  const double* rdx;     // 1 / dx
  const double* dt;      // time step
  const double* rmu;     // 1 / (2 mu)
  const double* u;       // velocity tables (FP64)
  const double* wt;
  const float* uf;       // FP32 copies
  const float* ul;       // u - uf: the FP32 velocities as hi + lo pairs
  const float* wtf;
  double* w;             // [cell][4] (3 used)
  double* prim;          // [cell][4]
  float* mc;             // [cell][8] FP32 Maxwellian coefficients of the cell's current prim
                         // (SegMax: rn, U hi, lambda, K / (2 lambda), U lo), kept with prim
  double* residual;      // [n][4]
  double* fw;            // [face][4] a single solve's face moments, null for ensembles: a step
                         // asked for its residual leaves its own, on the end faces too (with ghosts)
  // Per-step time step of a single solve (kb_step_cfl), null otherwise.  Step
  // number m has slot m mod 3: [slot] the CFL rate of the state before it,
  // [3 + slot] the time before it; then cfl, the end time, umax and the number
  // of steps taken.  A step reads its slot, collects the rate of its new state
  // in the next slot (atomic maximum over the segments) and clears the one
  // after, so no kernel stands between two steps and no host wait.
  double* clock;         // [10]
  int* active;           // [n] 1 while not converged
  int* status;
  // Segment k covers cells [seg_i0[k], seg_i0[k] + cells per segment) of
  // instance seg_b[k]; an instance's segments are consecutive from
  // seg_first[b] (nseg[b] of them)
  const int* seg_b;
  const int* seg_i0;
  const SegDesc* seg_d;  // FP32 kernel: the same and the instance's constants
  const int* seg_first;
  const int* nseg;
  double* respart;       // [segments][8] residual partial sums
  int nseg_all;          // segments of the current segment length
  int sst_max;           // largest shared-memory row stride of the batch (floats)
  int nu4_max;           // largest velocity count, rounded up to 4
  double K, gamma, omega, Pr, tol;
  double hg;             // 0.5 / (gamma - 1)
  float Kf, om1f, prf;   // K, 1 - omega and 0.8 (1 - Pr) in FP32
  double* mc64;          // [cell][4] FP64 Maxwellian coefficients of the cell's current prim
                         // (seg_coef64), kept with prim
  Pow64 tau_pow;         // lambda^(omega - 1) of the collision time
  int coll;
};

// The gas constants that follow from K, gamma, omega and Pr.
inline void seg_gas(BatchDev& d) {
  d.hg = 0.5 / (d.gamma - 1.0);
  d.Kf = float(d.K);
  d.om1f = float(1.0 - d.omega);
  d.prf = float(0.8 * (1.0 - d.Pr));
  d.tau_pow = pow64_of(d.omega - 1.0);
}

// Half the van Leer slope times dx from the differences a = q0 - qm and
// b = qp - q0, two at once: (a |b| + b |a|) / (|a| + |b| + eps) is
// 2 a b / (a + b +- eps) where a b > 0 and zero elsewhere (one reciprocal and
// one multiply, subnormals flushed).
__device__ __forceinline__ float2 bvl2(float2 a, float2 b, float eps) {
  const float2 p = p2mul(a, b), d = p2add(a, b);
  const float2 e = p2add(d, make_float2(copysignf(eps, d.x), copysignf(eps, d.y)));
  float rx, ry;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(e.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ry) : "f"(e.y));
  return p2mul(make_float2(fmaxf(p.x, 0.f), fmaxf(p.y, 0.f)), make_float2(rx, ry));
}

// 1D slope rule: van Leer everywhere inside when ghosts exist, boundary cells
// flat without ghosts (src/Solver/solver_reconstruction.jl:101-153).
__device__ __forceinline__ int brule(int i, int nx, int ng) {
  if (i < 0 || i >= nx) return 0;
  if (ng == 0 && (i == 0 || i == nx - 1)) return 0;
  return 1;
}

// e^x on the MUFU unit (2^(x log2 e), results below 2^-126 flushed to zero)
__device__ __forceinline__ float fexp(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}

// The FP32 Maxwellian of the segment kernel's relaxation and of the
// device-built equilibrium state (kb_batch_init_equilibrium, kb_pool_add):
// rn 2^(-lambda du^2 log2 e) with du = (u - U_hi) + (u_lo - U_lo).  Both
// use this one function, so a uniform equilibrium state is an exact fixed
// point of the FP32 update: fixed boundary cells and the cells next to them
// then agree bit for bit, and no FP32 rounding drift enters the FP64 w
// there (which, at high Mach number, the kinetic energy would amplify in T).
__device__ __forceinline__ float seg_maxwell(float u, float ulo, float rn, float Uh, float Ul,
                                             float lam) {
  const float du = (u - Uh) + (ulo - Ul);
  return rn * fexp(-lam * du * du);
}

// Two at once, of the difference du and -lambda (the same roundings)
__device__ __forceinline__ float2 seg_maxwell2(float2 du, float2 rn, float2 nlam) {
  const float2 x = p2mul(p2mul(p2mul(nlam, du), du), p2s(1.4426950408889634f));
  float2 y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
  return p2mul(rn, y);
}

// FP32 coefficients of one cell's Maxwellian from its FP64 prim [rho, U,
// lambda]: density factor rn = rho sqrt(lambda / pi), U as an FP32 pair,
// lambda, K / (2 lambda), each formed in FP64 and rounded once.
struct SegMax {
  float rn, Uh, Ul, lam, cB;
  __device__ __forceinline__ void set(const double* p, double K) {
    rn = f32_of(p[0] * sqrt64(p[2] * (1.0 / PI)));
    Uh = f32_of(p[1]);
    Ul = f32_of(p[1] - f64_of(Uh));
    lam = f32_of(p[2]);
    cB = f32_of((0.5 * K) * rcp64(p[2]));
  }
};

// The cell's FP32 Maxwellian coefficients into B.mc (kept with its prim).
__device__ __forceinline__ void seg_store_coef(const BatchDev& B, long cell, const SegMax& m) {
  float4* mcc = (float4*)(B.mc + cell * 8);
  mcc[0] = make_float4(m.rn, m.Uh, m.lam, m.cB);
  mcc[1] = make_float4(m.Ul, 0.f, 0.f, 0.f);
}

// Equilibrium h, b of cell c (0-based incl. ghosts) of instance b from the cell's
// coefficients (B.mc) into the FP32 buffers (init_fvm,
// src/Solver/solver_init.jl:119-141); row padding zero.  H0, B0: the buffer the
// next step reads; the other one takes what no step writes, ghost cells and
// padding.
__device__ __forceinline__ void seg_init_cell(const BatchDev& B, int b, int c, float* H0, float* B0,
                                              float* H1, float* B1) {
  const float4* mc = (const float4*)(B.mc + (B.cell_off[b] + c) * 8);
  const float4 m = mc[0];
  const float Ul = mc[1].x;
  const int nu = B.nu[b], ns = B.nus[b], ng = B.ng[b];
  const bool ghost = c < ng || c >= ng + B.nx[b];
  const long e = B.elem_off[b] + (long)c * ns;
  const float* uf = B.uf + B.vel_off[b];
  const float* ul = B.ul + B.vel_off[b];
  for (int v = threadIdx.x; v < ns; v += blockDim.x) {
    float hv = 0.f, bv = 0.f;
    if (v < nu) {
      hv = seg_maxwell(uf[v], ul[v], m.x, m.y, Ul, m.z);
      bv = hv * m.w;
    }
    H0[e + v] = hv;
    B0[e + v] = bv;
    if (ghost || v >= nu) {
      H1[e + v] = hv;
      B1[e + v] = bv;
    }
  }
}

// ---- per-step time step (BatchDev::clock)
struct SegClock {
  double dt, t;
  bool stop;  // the end time is reached: the state is carried over
  bool last;  // this step reaches it: its residual and face moments are kept
};
// timestep (src/Solver/solver_main.jl:240-288) from the collected rate
__device__ __forceinline__ SegClock seg_clock(const BatchDev& B, int slot) {
  SegClock c;
  const double tend = B.clock[7];
  c.t = B.clock[3 + slot];
  c.dt = B.clock[6] / B.clock[slot];
  c.dt = c.dt < tend - c.t ? c.dt : tend - c.t;
  const double end = tend - 1e-14 * fabs(tend);
  c.stop = !(c.t < end) || !(c.dt > 0.0);
  c.last = !(c.t + c.dt < end);
  return c;
}
// by one thread of the launch
__device__ __forceinline__ void seg_clock_next(const BatchDev& B, int slot, const SegClock& c) {
  const int nx = (slot + 1) % 3, clear = (slot + 2) % 3;
  B.clock[3 + nx] = c.stop ? c.t : c.t + c.dt;
  if (c.stop) B.clock[nx] = B.clock[slot];
  else B.clock[9] += 1.0;
  B.clock[clear] = 0.0;
}
__device__ __forceinline__ double seg_rate(const BatchDev& B, const double* p, double rdx) {
  return (fmax(B.clock[8], fabs(p[1])) + sqrt64((0.5 * B.gamma) * rcp64(p[2]))) * rdx;
}
// The rate of a state that no step may follow (not physical, or a wait that gave
// up): the next step's dt is 0, and the state is carried over from there.
__device__ __forceinline__ double seg_no_rate() { return __hiloint2double(0x7ff00000, 0); }
__device__ __forceinline__ void seg_clock_max(const BatchDev& B, int slot, double rate) {
  atomicMax((unsigned long long*)(B.clock + (slot + 1) % 3), (unsigned long long)__double_as_longlong(rate));
}
// The largest rate of a segment's cells (`rate`: the stepped cell of this
// lane) and of the fixed ends among them into the next slot; one warp.  Rates
// are positive, so their bits order like unsigned integers.
__device__ __forceinline__ void seg_clock_rate(const BatchDev& B, int slot, double rate, long c0, int ng,
                                               int i0, int i1, int nx, double rdx, int lane) {
  if (i0 == 0 && lane == 0) rate = fmax(rate, seg_rate(B, B.prim + (c0 + ng) * 4, rdx));
  if (i1 == nx && lane == 1) rate = fmax(rate, seg_rate(B, B.prim + (c0 + nx - 1 + ng) * 4, rdx));
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) rate = fmax(rate, __shfl_xor_sync(0xffffffffu, rate, o));
  if (lane == 0) seg_clock_max(B, slot, rate);
}

// ---- FP32 form: one CTA per segment of SEG cells, the whole step fused.
// In 1D an instance has at most 256 velocities, so a segment's stencil window
// (SEG + 4 cells x all velocities, h and b) fits in shared memory: the face
// moments of the segment's faces, the new w / prim / tau of its cells and
// the pointwise update all need only the old state inside that window, so
// the step is one pass over HBM (each value read once, plus a 2-cell halo on
// each side, and written once).  The window arrives by bulk async copies, one
// per row, into rows whose stride is = 16 (mod 32) floats so that the face
// threads read without bank conflicts.  Per-instance residuals are summed
// by k_batch_seg_res after the step, in segment order (deterministic).
//
// What bounds it: instruction issue.  512 shock structures (115,000 cells of 48
// to 200 velocities, 210 MB a step, 31 us of HBM) take 157 us a step: the face
// moments about 65 (two thirds of it the exact sums), the pointwise update 54,
// the FP64 cell warp 18, the window's latency the rest.  164 us with the clock of
// single solves in the same kernel, 189 before packed
// pairs, one descriptor load in front of the window (five dependent ones took
// 6,200 of a CTA's 36,000 cycles), sums merged by shuffles instead of by the
// cell warp, and two chunks of cells per thread instead of one velocity per
// thread (half the threads idle at 64 velocities).  At most 96 registers, five
// CTAs per multiprocessor: 178 us with 80 (spills), 195 with 120 (four CTAs).
constexpr int SEG_MAXNU = 256;
constexpr int SEG_CC = 7;  // float4 coefficient blocks per pair of cells
__host__ __device__ inline int seg_stride(int nus) { return (nus + 15) / 32 * 32 + 16; }
// Thread mapping of a segment CTA of SEG cells and T threads: a group of FT
// threads, a power of two, for each of the SEG + 1 faces in the face-moment
// phase (its sums are merged by shuffles); then one warp with a lane per cell;
// then one velocity and two chunks of cells per thread.
template <int SEG, int T>
struct SegShape {
  static constexpr int ROWS = SEG + 4;  // window cells
  static constexpr int FT = T / (SEG + 1);
  static_assert(SEG <= 31 && (SEG + 1) % 4 == 0 && T >= 64 && FT * (SEG + 1) == T && FT >= 4 && FT <= 32 &&
                    (FT & (FT - 1)) == 0,
                "segment shape");
};
// Dynamic shared memory of a segment CTA, sized by the batch's largest row
// stride and velocity count: h and b windows, velocity tables (hi, lo,
// weight), fw, the old w of the stepped cells, the coefficients of the cell
// pairs, the old Maxwellian coefficients and the heat fluxes.
template <int SEG, int T>
__host__ __device__ inline int seg_smem(int sst_max, int nu4_max) {
  return 2 * (SEG + 4) * sst_max * 4 + 3 * nu4_max * 4 + (SEG + 1) / 2 * SEG_CC * 16 + SEG * 32 +
         (SEG + 1) * 3 * 8 + SEG * 3 * 8 + (SEG + 1) * 4;
}
template <int SEG, int T>
__host__ __device__ inline int seg_smem_max() {
  return seg_smem<SEG, T>(seg_stride((SEG_MAXNU + 3) / 4 * 4), SEG_MAXNU);
}

// Sums of 4 values over a group of FT lanes: two levels that halve the values
// a lane carries, then plain ones.  Lane q of the group returns the total of
// value q / (FT / 4), merged in a fixed order.
template <int FT>
__device__ __forceinline__ DF seg_sums(DF (&x)[4], int lane) {
  DF y[2];
  const bool u1 = lane & (FT / 2), u0 = lane & (FT / 4);
#pragma unroll
  for (int k = 0; k < 2; ++k) y[k] = df_merge(u1 ? x[2 + k] : x[k], df_shfl_xor(u1 ? x[k] : x[2 + k], FT / 2));
  DF z = df_merge(u0 ? y[1] : y[0], df_shfl_xor(u0 ? y[0] : y[1], FT / 4));
#pragma unroll
  for (int m = FT / 8; m >= 1; m >>= 1) z = df_merge(z, df_shfl_xor(z, m));
  return z;
}

// Relaxation factors of a single solve's cell, each rounded once to FP32:
// dtt = dt / tau, tau = 2 mu lambda^(1 - omega) / rho (the power in FP32), and
// 1 / (1 + dtt) of the rounded dtt, so that their product is dtt / (1 + dtt) also
// where dtt is large; from dtm = dt / (2 mu) and om1 = omega - 1
__device__ __forceinline__ void seg_relax(double dtm, double rho, float lam, float om1, float& dtt, float& i1t) {
  dtt = f32_of(dtm * rho * f64_of(powf(lam, om1)));
  // 1 / (1 + dtt): the sum as s + e exactly, its reciprocal corrected by one
  // Newton step (FP32: the FP64 form holds the cell warp 0.2 us longer)
  const float s = 1.f + dtt, b = s - 1.f, e = (1.f - (s - b)) + (dtt - b), r = __frcp_rn(s);
  i1t = fmaf(r, fmaf(-s, r, 1.f) - e * r, r);
}
// Its Shakhov factor 0.8 (1 - Pr) lambda^2 q / rho (of the old state)
__device__ __forceinline__ float seg_heat(double c, double lam, double rho, double q) {
  return f32_of(c * (lam * lam) * rcp64(rho) * q);
}
// A term of the residual in its sum's precision, and the sum in FP64
template <typename R> __device__ __forceinline__ R seg_res_term(double x);
template <> __device__ __forceinline__ double seg_res_term<double>(double x) { return x; }
template <> __device__ __forceinline__ float seg_res_term<float>(double x) { return f32_of(x); }
__device__ __forceinline__ double seg_res_sum(double x) { return x; }
__device__ __forceinline__ double seg_res_sum(float x) { return f64_of(x); }

// Segment k covers cells [seg_i0[k], seg_i0[k] + SEG) of instance seg_b[k].
// A CTA takes segments k = blockIdx.x, blockIdx.x + gridDim.x, ...: one
// segment each when the grid has a CTA per segment, or a persistent loop
// when the grid is the number of CTAs that fit on the GPU at once.
// res: the residual's partial sums are wanted.  ONE: the form of a single
// solve, with its own time step (slot: BatchDev::clock, -1: B.dt) and face moments
// (BatchDev::fw); a form of its own, because they cost the ensembles' 1.6 %.
template <int SEG, int SEG_T, bool ONE = false>
__global__ void __launch_bounds__(SEG_T, SEG < 7 ? 1 : 20 * 32 / SEG_T)
    k_batch_seg(BatchDev B, const float* Hin, const float* Bin,
                float* __restrict__ Hout, float* __restrict__ Bout, int slot, int res) {
  using SH = SegShape<SEG, SEG_T>;
  constexpr int SEG_ROWS = SH::ROWS;
  constexpr int FT = SH::FT;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ unsigned long long bar;
  __shared__ float sconst[2];  // T3, T4
  __shared__ int sflag[2];     // (ONE) the step is past the end; its residual and face moments are kept
  __shared__ double sdtm;      // (ONE) dt / (2 mu)
  // An FP64 instruction holds a quarter of the multiprocessor for 64 cycles
  // whatever its active lanes, so the FP64 cell phase is one warp's, written
  // for few instructions (about 30; the divisions, conversions and compares
  // of the plain form took 140), and which warp it is changes from segment to
  // segment: a CTA's warp number decides its quarter, and one fixed warp would
  // queue every resident CTA's cell phase on the same one.
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_async_smem();
  }
  __syncthreads();
  unsigned phase = 0;  // completed window copies of this CTA (mbarrier parity)
  for (int k = blockIdx.x; k < B.nseg_all; k += gridDim.x) {
  const SegDesc sd = B.seg_d[k];
  const int b = sd.b, i0 = sd.i0, nx = sd.nx, ng = sd.ng, nu = sd.nu, ns = sd.ns;
  const int i1 = min(i0 + SEG, nx);
  const long c0 = sd.c0;
  const float* Hi = Hin + sd.e0;
  const float* Bi = Bin + sd.e0;
  float* Ho = Hout + sd.e0;
  float* Bo = Bout + sd.e0;
  const int sst = seg_stride(ns);
  // window rows r0 .. r1-1 (cells incl. ghosts), smem row = cell - r0
  const int r0 = max(i0 - 2, -ng), r1 = min(i1 + 2, nx + ng), nrow = r1 - r0;
  float* sH = (float*)sm;
  float* sB = sH + SEG_ROWS * B.sst_max;
  float* sU = sB + SEG_ROWS * B.sst_max;
  float* sW = sU + B.nu4_max;
  float* sUl = sW + B.nu4_max;  // low parts of the velocities
  // [(SEG + 1) / 2][SEG_CC] coefficients of cell pairs
  float4* scc = (float4*)(sUl + B.nu4_max);
  float4* smc = scc + (SEG + 1) / 2 * SEG_CC;  // [SEG][2] see B.mc
  double* sfw = (double*)(smc + SEG * 2);      // [SEG + 1][3]
  double* swo = sfw + (SEG + 1) * 3;           // [SEG][3] w
  float* sq = (float*)(swo + SEG * 3);         // [SEG + 1] heat flux of the cell right of the face
  // up to here only what no step writes
  pdl_wait();
  pdl_next();
  // The window first: it is on its way while the rest is read (one load deep).
  if (tid < 32) {
    if (lane == 0) mbar_expect(&bar, 2u * nrow * ns * 4u);
    __syncwarp();
    for (int r = lane; r < 2 * nrow; r += 32) {
      const int row = r >> 1;
      const float* src = ((r & 1) ? Bi : Hi) + (long)(r0 + row + ng) * ns;
      float* dst = ((r & 1) ? sB : sH) + row * sst;
      bulk_g2s(dst, src, (unsigned)ns * 4u, &bar);
    }
  }
  const bool skip = !B.active[b];
  const int ca = max(i0, 1), cb = min(i1, nx - 1);  // stepped cells [ca, cb); may be none
  const int ncell = cb - ca;
  for (int v = tid; v < ns; v += SEG_T) {  // zero weight up to the row's end
    sU[v] = v < nu ? B.uf[sd.vo + v] : 0.f;
    sUl[v] = v < nu ? B.ul[sd.vo + v] : 0.f;
    sW[v] = v < nu ? B.wtf[sd.vo + v] : 0.f;
  }
  if (tid < ncell) {  // old w and Maxwellian coefficients of the stepped cells
    const long c = c0 + ca + tid + ng;
    swo[tid * 3 + 0] = B.w[c * 4 + 0];
    swo[tid * 3 + 1] = B.w[c * 4 + 1];
    swo[tid * 3 + 2] = B.w[c * 4 + 2];
    smc[tid * 2] = ((const float4*)(B.mc + c * 8))[0];
    smc[tid * 2 + 1] = ((const float4*)(B.mc + c * 8))[1];
    if (ONE) *(double*)&smc[tid * 2 + 1].z = B.prim[c * 4 + 2];
  }
  if (tid == SEG_T - 1) {
    double dt0 = B.dt[b];
    if (ONE) {
      SegClock c = {dt0, 0.0, false, false};
      if (slot >= 0) {
        c = seg_clock(B, slot);
        if (k == 0) seg_clock_next(B, slot, c);
      }
      dt0 = c.dt;
      sdtm = c.dt * B.rmu[b];
      sflag[0] = c.stop;
      sflag[1] = res || c.last;
    }
    sconst[0] = f32_of(dt0);
    sconst[1] = f32_of(0.5 * dt0 * dt0 * sd.rdx);
  }
  // one thread waits for the window; the others wait at the CTA barrier
  const bool ok = tid == 0 ? mbar_wait(&bar, phase & 1) : true;
  if (__syncthreads_or(!ok)) {  // CTA-uniform: bounded clean-up, then leave
    if (tid == 0) {
      atomicOr(B.status, 2);
      if (ONE && slot >= 0) seg_clock_max(B, slot, seg_no_rate());
      mbar_wait(&bar, phase & 1);
    }
    return;
  }
  ++phase;
  const int dB = SEG_ROWS * B.sst_max;  // from a value of h to the same of b
  const bool want = ONE ? sflag[1] != 0 : res != 0;
  if (skip || (ONE && sflag[0])) {  // converged or past the end: carry this segment's cells over
    for (int i = i0; i < i1; ++i)
      for (int v = tid; v < ns; v += SEG_T) {
        Ho[(long)(i + ng) * ns + v] = sH[(i - r0) * sst + v];
        Bo[(long)(i + ng) * ns + v] = sH[(i - r0) * sst + v + dB];
      }
    __syncthreads();  // the window is reused by the next segment
    continue;  // CTA-uniform
  }
  const int fa = ca;  // faces fa .. fa + ncell: the left faces of the stepped cells and the last one's right face
  const float epsd = sd.epsd;
  const float T3 = sconst[0], T4 = sconst[1];
  const bool shak = B.coll == COLL_SHAKHOV;
  // The pointwise phase's split: a thread takes one velocity and two chunks of
  // L cells in packed arithmetic.  Chunks of ceil(ncell / 2, 4, 8) cells: the
  // one with the least rounds of the CTA times (cells + half a cell for the
  // chunk's first face), so that 48 velocities fill 128 threads as well as 128
  // or 160 do.
  int L = (ncell + 1) >> 1, ngrp = 1;
  {
    int best = ((nu + SEG_T - 1) / SEG_T) * (2 * L + 1);
#pragma unroll
    for (int lg = 2; (1 << lg) <= (SEG < 7 ? SEG + 1 : 8); ++lg) {
      const int l = (ncell + (1 << lg) - 1) >> lg, g = 1 << (lg - 1);
      const int c = ((nu * g + SEG_T - 1) / SEG_T) * (2 * l + 1);
      if (c < best) {
        best = c;
        L = l;
        ngrp = g;
      }
    }
  }

  // ---- face moments of those faces and heat flux of the cells right of
  // them: FT threads per face (velocity pairs q mod FT).  A half-warp reads 16
  // pairs: rows of 16 (mod 32) floats put two faces' pairs on all the banks.
  {
    const int j = tid / FT, q = tid % FT;
    // the faces, then the ends' for BatchDev::fw (a segment with an end steps a
    // cell less, so a group of threads is free for it)
    const bool keep = ONE && want;
    const int end0 = keep && ng > 0 && i0 == 0, end1 = keep && ng > 0 && i1 == nx;
    const int f = j <= ncell ? fa + j : (j == ncell + 1 && end0 ? 0 : nx);
    const bool live = j <= ncell + end0 + end1;
    // Each moment term enters as an exact pair: the FP32 products w fh,
    // w fh u, w fh u^2, w fb with their rounding errors (FMA), added with
    // error-free sums (TwoSum), the two velocities in packed arithmetic.  In a
    // supersonic flow the energy flux is large and the flux difference between
    // a cell's two faces small, so FP32 rounding of the terms or of running
    // partial sums would enter w as a bias of relative size ~1e-7 of the flux
    // every step -- amplified in T = 1 / (2 lambda) by the kinetic-to-thermal
    // energy ratio (~35 at Mach 8), it grew to 1e-5 of T within a few hundred
    // steps.
    const float2 zero = make_float2(0.f, 0.f);
    float2 s0 = zero, s1 = zero, s2 = zero, sb = zero, sq2 = zero;  // sums
    float2 l0 = zero, l1 = zero, l2 = zero, lb = zero, lq = zero;  // their rounding errors
    float2 e0 = zero, e1 = zero, e2 = zero;                        // and the products'
    if (live) {
      const int iL = f - 1, iR = f;
      const bool vlL = brule(iL, nx, ng) == 1, vlR = brule(iR, nx, ng) == 1;
      // window offsets of the three cells around the upwind one (clamped where
      // the slope rule reads no neighbour): iL's for u >= 0, iR's otherwise
      const int oL = (iL - r0) * sst, oR = (iR - r0) * sst;
      const int oLL = (max(iL - 1, r0) - r0) * sst, oRR = (min(iR + 1, r1 - 1) - r0) * sst;
      const bool hf = shak && j < ncell;
      const float Uh = hf ? smc[j * 2].y : 0.f, Ul = hf ? smc[j * 2 + 1].x : 0.f;
      float2 pq = zero;  // heat-flux terms, eight at a time
      int it = 0;
      for (int v = 2 * q; v < nu; v += 2 * FT, ++it) {
        const float2 u = *(const float2*)(sU + v), w = *(const float2*)(sW + v);
        const bool px = u.x >= 0.f, py = u.y >= 0.f;
        const float* m = sH + (px ? oLL : oL) + v;
        const float* c = sH + (px ? oL : oR) + v;
        const float* r = sH + (px ? oR : oRR) + v;
        float2 hm = *(const float2*)m, h0 = *(const float2*)c, hp = *(const float2*)r;
        float2 bm = *(const float2*)(m + dB), b0 = *(const float2*)(c + dB), bp = *(const float2*)(r + dB);
        if (px != py) {  // the one pair that straddles u = 0
          m = sH + (py ? oLL : oL) + v + 1;
          c = sH + (py ? oL : oR) + v + 1;
          r = sH + (py ? oR : oRR) + v + 1;
          hm.y = *m;
          h0.y = *c;
          hp.y = *r;
          bm.y = m[dB];
          b0.y = c[dB];
          bp.y = r[dB];
        }
        const float2 sh = bvl2(p2sub(h0, hm), p2sub(hp, h0), epsd), sv = bvl2(p2sub(b0, bm), p2sub(bp, b0), epsd);
        // T3 u (h0 +- s / 2) - T4 u^2 s = T3 u h0 + |u| (T3 / 2 - T4 |u|) s
        const float2 au = make_float2(fabsf(u.x), fabsf(u.y));
        const float2 Tu = p2mul(p2s(T3), u);
        float2 cs = p2mul(au, p2fma(p2s(-2.f * T4), au, p2s(T3)));
        cs.x = (px ? vlL : vlR) ? cs.x : 0.f;
        cs.y = (py ? vlL : vlR) ? cs.y : 0.f;
        const float2 fh = p2fma(Tu, h0, p2mul(cs, sh)), fbv = p2fma(Tu, b0, p2mul(cs, sv));
        // rounded products and, negated, their errors: w fh = t0 - n0 exactly
        const float2 nw = make_float2(-w.x, -w.y), nu2 = make_float2(-u.x, -u.y);
        const float2 t0 = p2mul(w, fh), n0 = p2fma(nw, fh, t0);
        const float2 tb = p2mul(w, fbv), nb = p2fma(nw, fbv, tb);
        const float2 t1 = p2mul(t0, u), n1 = p2fma(n0, u, p2fma(nu2, t0, t1));  // w fh u = t1 - n1
        const float2 t2 = p2mul(t1, u), n2 = p2add(p2fma(n1, u, p2fma(nu2, t1, t2)), nb);
        p2df_add(s0, l0, t0);
        p2df_add(s1, l1, t1);
        p2df_add(s2, l2, t2);
        p2df_add(sb, lb, tb);
        e0 = p2add(e0, n0);
        e1 = p2add(e1, n1);
        e2 = p2add(e2, n2);  // w (fh u^2 + fb) = t2 + tb - n2
        if (hf) {  // heat_flux 2F1V of cell iR: the row right of or at the upwind one
          const float2 ul = *(const float2*)(sUl + v);
          const float2 hc = make_float2(px ? hp.x : h0.x, py ? hp.y : h0.y);
          const float2 bc = make_float2(px ? bp.x : b0.x, py ? bp.y : b0.y);
          const float2 cu = p2add(p2sub(u, p2s(Uh)), p2sub(ul, p2s(Ul)));
          pq = p2fma(p2mul(w, cu), p2fma(p2mul(cu, cu), hc, bc), pq);
          if ((it & 7) == 7) {
            p2df_add(sq2, lq, pq);
            pq = zero;
          }
        }
      }
      p2df_add(sq2, lq, pq);
    }
    // merged over the face's threads in a fixed order: both segments that
    // share a face map its velocities to the same threads q, so they compute
    // bit-identical fw (conservation holds exactly)
    const auto fold = [](float2 s, float2 lo) {
      DF d;
      d.hi = s.x;
      d.lo = lo.x + lo.y;
      df_add(d, s.y);
      return d;
    };
    DF x[4] = {fold(s0, p2sub(l0, e0)), fold(s1, p2sub(l1, e1)), fold(s2, p2sub(p2add(l2, lb), e2)), fold(sq2, lq)};
    df_add(x[2], sb.x);
    df_add(x[2], sb.y);
    const DF t = seg_sums<FT>(x, lane);
    const int m = q / (FT / 4);
    if (q % (FT / 4) == 0) {
      const float half = m < 2 ? 1.f : 0.5f;
      if (m < 3) {
        const double S = f64_of(half * t.hi) + f64_of(half * t.lo);
        sfw[j * 3 + m] = S;
        if (keep && live && (f > i0 || f <= 1)) B.fw[(long)f * 4 + m] = S;  // (face i0: the segment's before)
      } else {
        sq[j] = half * (t.hi + t.lo);
        if (ONE && j < ncell) smc[j * 2 + 1].y = half * t.lo - (sq[j] - half * t.hi);
      }
    }
  }
  __syncthreads();  // face moments and heat fluxes in shared memory
  // Coefficient block n of cell ca + j: the cells of a pair sit side by side
  auto coef = [&](int j, int n) {
    const int g = j / (2 * L), r = j - 2 * L * g;
    const int hi = r >= L ? 1 : 0;
    return (float*)(scc + (g * L + r - hi * L) * SEG_CC) + 2 * n + hi;
  };
  // The cell warp: the FP64 cell update.
  const int role = (wid + (int)(((unsigned)k * 2654435761u) >> 29)) % (SEG_T / 32);
  if (ONE && role == 1 && shak && lane < ncell) {
    // the heat-flux factor (below) in FP64, beside the cell warp
    const double lo = *(const double*)&smc[lane * 2 + 1].z;
    const double q = f64_of(sq[lane]) + f64_of(smc[lane * 2 + 1].y);
    coef(lane, 0)[24] = seg_heat(0.8 * (1.0 - B.Pr), lo, swo[lane * 3], q);
  }
  if (role == 0) {
    double rate = 0.0;  // CFL rate of the cell's new state (slot >= 0)
    // ---- cell parameters of the stepped cells (one lane per cell, FP64)
    if (lane < ncell) {
      const double rdx = sd.rdx;
      const int i = ca + lane;
      const long c = c0 + i + ng;
      double* w = B.w + c * 4;
      double* p = B.prim + c * 4;
      const double* fL = sfw + lane * 3;
      const double* fR = fL + 3;
      double wn[3];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        wn[m] = fma(fL[m] - fR[m], rdx, swo[lane * 3 + m]);
        w[m] = wn[m];
      }
      // conserve_prim (src/Theory/theory_macro.jl:185-206), hg = 0.5 / (gamma - 1)
      double pn[3];
      const double rr0 = rcp64(wn[0]);
      pn[0] = wn[0];
      pn[1] = wn[1] * rr0;
      pn[2] = wn[0] * B.hg * rcp64(fma(-0.5 * wn[1], pn[1], wn[2]));
      p[0] = pn[0];
      p[1] = pn[1];
      p[2] = pn[2];
      if (ONE && slot >= 0) rate = seg_rate(B, pn, rdx);
      if (!pos64(pn[0]) || !pos64(pn[2])) {
        atomicOr(B.status, 1);
        rate = seg_no_rate();
      }
      // w, prim and q stay FP64; the coefficients below feed only the FP32
      // pointwise update.  The Maxwellian's density factor, U and lambda are
      // formed in FP64 and rounded once, and U is carried as an FP32 pair
      // (hi + lo) so that u - U is exact to FP32 rounding of the difference:
      // at high Mach the energy is mostly kinetic, and an FP32-rounded U or
      // density factor would bias the moments of the equilibrium by more
      // than the FP32 split form's 1e-5 budget in T.  tau only sets the
      // relaxation rate: FP32 in the ensembles, and in a single solve, as in the
      // general form, FP64 but for the power.
      SegMax mn;  // the new Maxwellian
      mn.set(pn, B.K);
      float dtt, i1t;
      if (ONE) {
        seg_relax(sdtm, pn[0], mn.lam, -B.om1f, dtt, i1t);
      } else {
        dtt = sconst[0] / (sd.mu2 * powf(mn.lam, B.om1f) / f32_of(pn[0]));
        i1t = 1.f / (1.f + dtt);
      }
      // the old Maxwellian's coefficients are the ones this cell's update
      // formed from the same prim one step earlier (or the set-up formed from
      // the initial prim): read instead of recomputed
      const float4 mo = smc[lane * 2];
      // new Maxwellian: density factor, U (hi, lo), -lambda, K / (2 lambda);
      // dt / tau, 1 / (1 + dt / tau); old Maxwellian (Shakhov): density factor,
      // U (hi, lo), -lambda, K / (2 lambda), and the heat-flux factor
      // 0.8 (1 - Pr) lambda^2 / rho q of the old state
      const float kc[13] = {mn.rn, mn.Uh, mn.Ul, -mn.lam, mn.cB, dtt, i1t,
                            mo.x,  mo.y,  smc[lane * 2 + 1].x, -mo.z, mo.w,
                            shak && !ONE ? B.prf * (mo.z * mo.z) / f32_of(swo[lane * 3]) * sq[lane] : 0.f};
      float* kp = coef(lane, 0);
#pragma unroll
      for (int n = 0; n < (ONE ? 12 : 13); ++n) kp[2 * n] = kc[n];
      seg_store_coef(B, c, mn);
    }
    if (want) {  // this segment's residual partial sums (k_batch_seg_res adds them up)
      // squares of FP64 differences: a convergence monitor that the ensembles sum
      // in FP32, a single solve in FP64
      using RR = typename std::conditional<ONE, double, float>::type;
      RR rr[6] = {0, 0, 0, 0, 0, 0};
      if (lane < ncell) {
        const double* w = B.w + (c0 + ca + lane + ng) * 4;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const double wn = w[m], dw = wn - swo[lane * 3 + m];
          rr[m] = seg_res_term<RR>(dw * dw);
          rr[3 + m] = seg_res_term<RR>(fabs(wn));
        }
      }
#pragma unroll
      for (int m = 0; m < 6; ++m) {
#pragma unroll
        for (int o = (SEG + 1) / 2; o >= 1; o >>= 1) rr[m] += __shfl_xor_sync(0xffffffffu, rr[m], o);
      }
      if (lane == 0) {
        double* pr = B.respart + (long)k * 8;
#pragma unroll
        for (int m = 0; m < 6; ++m) pr[m] = seg_res_sum(rr[m]);
      }
    }
    if (ONE && slot >= 0) seg_clock_rate(B, slot, rate, c0, ng, i0, i1, nx, sd.rdx, lane);
  }
  __syncthreads();  // cell coefficients ready for the pointwise update
  // ---- pointwise KFVS flux + relaxation: a thread marches two chunks of L
  // cells at its velocity, in packed arithmetic, each window row read once.
  // Every upwind cell of a segment away from ghost-less ends takes the van Leer
  // slope, so that form skips the per-face slope rule.
  for (int v = tid; v < nu; v += SEG_T) {  // fixed end cells keep their state
    if (i0 == 0) {
      Ho[(long)ng * ns + v] = sH[(0 - r0) * sst + v];
      Bo[(long)ng * ns + v] = sH[(0 - r0) * sst + v + dB];
    }
    if (i1 == nx) {
      Ho[(long)(nx - 1 + ng) * ns + v] = sH[(nx - 1 - r0) * sst + v];
      Bo[(long)(nx - 1 + ng) * ns + v] = sH[(nx - 1 - r0) * sst + v + dB];
    }
  }
  const float2 idx = p2s(f32_of(sd.rdx));
  const bool all_vl = ng > 0 || (ca >= 2 && cb <= nx - 2);
  auto pointwise = [&](auto vl_tag) {
    constexpr bool VL = decltype(vl_tag)::value;
    for (int it = tid; it < nu * ngrp; it += SEG_T) {
      int v = it, g = 0;
      for (; v >= nu; ++g) v -= nu;
      const int a0 = ca + 2 * L * g;                      // the chunks' first cells
      const int nA = min(L, cb - a0), nB = cb - (a0 + L);  // and numbers (nB may be below 1 or above L)
      if (nA <= 0) continue;
      const float u = sU[v], au = fabsf(u);
      const bool pos = u >= 0.f;
      const float2 Tu = p2s(T3 * u), cs = p2s(au * fmaf(-2.f * T4, au, T3));
      const float2 u2 = p2s(u), ul2 = p2s(sUl[v]);
      // the upwind cell of a chunk's first face and the rows around it; past
      // the window's ends (no slope there, or beyond the second chunk's last
      // cell) the row stays the end one
      const int cA = a0 - (pos ? 1 : 0), cB = cA + L;
      const int last = (r1 - 1 - r0) * sst;
      const float* hv = sH + v;
      int oA = (cA - r0) * sst, oB = min((cB - r0) * sst, last);
      const int mA = VL ? oA - sst : max(oA - sst, 0), mB = min((cB - 1 - r0) * sst, last);
      float2 hm = make_float2(hv[mA], hv[mB]), bm = make_float2(hv[mA + dB], hv[mB + dB]);
      float2 h0 = make_float2(hv[oA], hv[oB]), b0 = make_float2(hv[oA + dB], hv[oB + dB]);
      float2 dh = p2sub(h0, hm), db = p2sub(b0, bm);
      float2 hp, bp, dhp, dbp;
      // the flux out of the upwind cells (cA + k, cB + k); moves hp, bp one on
      auto face = [&](int k, float2& fh, float2& fb) {
        oA = VL ? oA + sst : min(oA + sst, last);
        oB = min(oB + sst, last);
        hp = make_float2(hv[oA], hv[oB]);
        bp = make_float2(hv[oA + dB], hv[oB + dB]);
        dhp = p2sub(hp, h0);
        dbp = p2sub(bp, b0);
        float2 c = cs;
        if (!VL) {
          c.x = brule(cA + k, nx, ng) == 1 ? c.x : 0.f;
          c.y = brule(cB + k, nx, ng) == 1 ? c.y : 0.f;
        }
        fh = p2fma(Tu, h0, p2mul(c, bvl2(dh, dhp, epsd)));
        fb = p2fma(Tu, b0, p2mul(c, bvl2(db, dbp, epsd)));
      };
      float2 fhL, fbL;
      face(0, fhL, fbL);
      long o = (long)(a0 + ng) * ns + v;
      const long oL = (long)L * ns;
      const float4* kc = scc + g * L * SEG_CC;
      for (int k = 0; k < nA; ++k, o += ns, kc += SEG_CC) {
        hm = h0;
        bm = b0;
        h0 = hp;
        b0 = bp;
        dh = dhp;
        db = dbp;
        float2 fhR, fbR;
        face(k + 1, fhR, fbR);
        // the cells themselves: upwind of the right face where u >= 0, of the
        // left one otherwise
        const float2 hc = make_float2(pos ? h0.x : hm.x, pos ? h0.y : hm.y);
        const float2 bc = make_float2(pos ? b0.x : bm.x, pos ? b0.y : bm.y);
        const float4 k0 = kc[0], k1 = kc[1], k2 = kc[2], k3 = kc[3];
        const float2 du = p2add(p2sub(u2, make_float2(k0.z, k0.w)), p2sub(ul2, make_float2(k1.x, k1.y)));
        const float2 M = seg_maxwell2(du, make_float2(k0.x, k0.y), make_float2(k1.z, k1.w));
        float2 MH = M, MB = p2mul(M, make_float2(k2.x, k2.y));
        if (shak) {
          const float4 k4 = kc[4], k5 = kc[5];
          const float2 qf = *(const float2*)(kc + 6);
          const float2 ou = p2add(p2sub(u2, make_float2(k4.x, k4.y)), p2sub(ul2, make_float2(k4.z, k4.w)));
          const float2 nl = make_float2(k5.x, k5.y);
          const float2 OH = seg_maxwell2(ou, make_float2(k3.z, k3.w), nl);
          const float2 y = p2mul(p2mul(nl, ou), ou);  // -lambda ou^2
          const float2 cq = p2mul(p2mul(qf, ou), OH);
          MH = p2fma(cq, p2fma(y, p2s(-2.f), p2s(B.Kf - 5.f)), MH);
          MB = p2fma(p2mul(cq, make_float2(k5.z, k5.w)), p2fma(y, p2s(-2.f), p2s(B.Kf - 3.f)), MB);
        }
        // (h + div + dt/tau MH) / (1 + dt/tau) written as a correction of h,
        // so that an equilibrium cell (MH == h, div == 0) stays bit-exact
        const float2 dt2 = make_float2(k2.z, k2.w), i1k = make_float2(k3.x, k3.y);
        const float2 nh = p2fma(p2fma(p2sub(fhL, fhR), idx, p2mul(dt2, p2sub(MH, hc))), i1k, hc);
        const float2 nb = p2fma(p2fma(p2sub(fbL, fbR), idx, p2mul(dt2, p2sub(MB, bc))), i1k, bc);
        Ho[o] = nh.x;
        Bo[o] = nb.x;
        if (k < nB) {
          Ho[o + oL] = nh.y;
          Bo[o + oL] = nb.y;
        }
        fhL = fhR;
        fbL = fbR;
      }
    }
  };
  if (all_vl) pointwise(std::true_type{});
  else pointwise(std::false_type{});
  __syncthreads();  // the window and coefficients are reused by the next segment
  }
}


// One compiled shape of the segment kernel.
struct SegVariant {
  int seg, threads;               // the shape's name: faces per CTA, threads
  int cells;                      // cells per segment
  const void* fn;                 // k_batch_seg<seg, threads>
  int (*smem)(int sst_max, int nu4_max);
  int smem_max;
};
// The compiled shapes (kb_batch.cu).
const std::vector<SegVariant>& seg_variants();
void seg_variants_a(std::vector<SegVariant>& out);
void seg_variants_b(std::vector<SegVariant>& out);

}  // namespace kb
