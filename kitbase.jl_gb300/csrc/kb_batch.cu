// kb_batch.cu -- many independent 1D2F1V solves (uneven cell counts and
// velocity grids) advanced by one fused kernel launch per time step.
//
// Ragged layout: instance b owns cells [cell_off[b], cell_off[b] + nxt[b])
// (ghosts included) and a velocity table at vel_off[b] of length nu[b]; its
// distributions start at elem_off[b] in the flat h / b arrays and are
// [cell][nus[b]] (velocity fastest, rows padded to a multiple of 4 values so
// every row starts 16-byte aligned for bulk copies).  A CTA fuses the whole
// step of one segment of one instance: face moments and old heat flux, cell
// parameters (w, prim, tau), pointwise KFVS flux + BGK / Shakhov relaxation,
// in one pass over HBM (k_batch_seg in FP32, k_batch_seg64 in FP64);
// k_batch_seg_res forms each instance's residual and convergence flag from its
// segments' partial sums.
// Covers the configuration of the batched shock-structure ensemble: KFVS,
// BGK or Shakhov, fixed boundaries, van Leer, up to 256 velocities.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/kitgpu.h"
#include "kb_batch.cuh"
#include "kb_batch64.cuh"

namespace kb {

// Residual of each active instance of the segment form
// (src/Solver/solver_update.jl:86-88) and its convergence flag.  One warp per
// instance: lane l adds the partial sums of segments l, l + 32, ... in order,
// then a fixed shuffle tree combines the lanes (deterministic).  Launched
// after k_batch_seg on the same stream, so no segment CTA waits on a fence or
// an atomic counter of the others.
__global__ void k_batch_seg_res(BatchDev B) {
  const int b = (int)((blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  pdl_wait();
  pdl_next();
  if (b >= B.n || !B.active[b]) return;  // warp-uniform
  double t[6] = {0, 0, 0, 0, 0, 0};
  const int s0 = B.seg_first[b], s1 = s0 + B.nseg[b];
  for (int sgi = s0 + lane; sgi < s1; sgi += 32)
    for (int m = 0; m < 6; ++m) t[m] += B.respart[(long)sgi * 8 + m];
#pragma unroll
  for (int m = 0; m < 6; ++m) t[m] = warp_sum(t[m]);
  if (lane == 0) {
    double mx = 0.0;
    for (int m = 0; m < 3; ++m) {
      const double r = sqrt(t[m] * B.nx[b]) / (t[3 + m] + 1.e-7);
      B.residual[b * 4 + m] = r;
      mx = fmax(mx, r);
    }
    if (mx < B.tol) B.active[b] = 0;
  }
}

void seg_res_launch(const BatchDev& B, cudaStream_t st) {
  void* args[] = {(void*)&B};
  launch_after((const void*)k_batch_seg_res, dim3((unsigned)((B.n + 3) / 4)), dim3(128), 0, st, args);
}

__global__ void k_batch_timestep(BatchDev B, const double* umax, double cfl, double* dt_out,
                                 int b0 = 0) {
  const int b = b0 + blockIdx.x;
  __shared__ double red[256];
  const int nx = B.nx[b], ng = B.ng[b];
  double m = 0.0;
  for (int i = threadIdx.x; i < nx; i += blockDim.x) {
    const double* p = B.prim + (B.cell_off[b] + i + ng) * 4;
    const double sos = sqrt64((0.5 * B.gamma) * rcp64(p[2]));
    m = fmax(m, (fmax(umax[b], fabs(p[1])) + sos) * B.rdx[b]);
  }
  red[threadIdx.x] = m;
  __syncthreads();
  for (int s = blockDim.x / 2; s >= 1; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) dt_out[b] = cfl / red[0];
}

// Equilibrium h, b of instances' cells into both FP32 buffers with the
// relaxation's own FP32 Maxwellian (seg_init_cell): blockIdx.y = instance
// b0 + y, blockIdx.x = cell.
__global__ void k_batch_init_eq32(BatchDev B, int b0, float* H0, float* B0, float* H1, float* B1) {
  const int b = b0 + blockIdx.y;
  if ((int)blockIdx.x >= B.nx[b] + 2 * B.ng[b]) return;
  seg_init_cell(B, b, blockIdx.x, H0, B0, H1, B1);
}

// FP32 Maxwellian coefficients of every cell from its prim (after a host upload
// of prim, and for the equilibrium start): blockIdx.y = instance b0 + y, one
// thread per cell.
__global__ void k_batch_mcache(BatchDev B, int b0) {
  const int b = b0 + blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= B.nx[b] + 2 * B.ng[b]) return;
  const long cell = B.cell_off[b] + c;
  SegMax m;
  m.set(B.prim + cell * 4, B.K);
  seg_store_coef(B, cell, m);
}

void seg_mcache_launch(const BatchDev& B, int n, int max_cells, cudaStream_t st, int b0) {
  k_batch_mcache<<<dim3((unsigned)((max_cells + 127) / 128), (unsigned)n), 128, 0, st>>>(B, b0);
}

// FP64 form: h = maxwellian(u, prim), b = h K / (2 lambda) in FP64
// (src/Theory/theory_equilibrium.jl:8-13) into both buffers.
__global__ void k_batch_init_eq64(BatchDev B, double* H0, double* B0, double* H1, double* B1) {
  const int b = blockIdx.y;
  if ((int)blockIdx.x >= B.nx[b] + 2 * B.ng[b]) return;
  const double* p = B.prim + (B.cell_off[b] + blockIdx.x) * 4;
  const double rn = p[0] * sqrt(p[2] / PI), cB = B.K / (2.0 * p[2]);
  const int nu = B.nu[b], ns = B.nus[b];
  const long e = B.elem_off[b] + (long)blockIdx.x * ns;
  const double* u = B.u + B.vel_off[b];
  for (int v = threadIdx.x; v < ns; v += blockDim.x) {
    double hv = 0.0, bv = 0.0;
    if (v < nu) {
      const double du = u[v] - p[1];
      hv = rn * exp(-p[2] * du * du);
      bv = hv * cB;
    }
    H0[e + v] = hv;
    B0[e + v] = bv;
    H1[e + v] = hv;
    B1[e + v] = bv;
  }
}

template <typename R>
__global__ void k_batch_convert(R* dst, const double* src, long n) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = (R)src[t];
}
template <typename R>
__global__ void k_batch_back(double* dst, const R* src, long n) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) dst[t] = (double)src[t];
}

}  // namespace kb

// ---------------------------------------------------------------- C ABI

struct kb_batch {
  kb::BatchDev d;
  int prec = 0;
  int n = 0;
  long ncell = 0, nelem = 0, nvel = 0;
  void* h[2] = {nullptr, nullptr};
  void* bq[2] = {nullptr, nullptr};
  int cur = 0;
  cudaStream_t stream = nullptr;
  std::vector<void*> allocs;
  std::vector<int> nx, ng, nu, nus;
  std::vector<double> dx, mu;
  std::vector<long> vel_off_h;
  std::vector<long> cell_off, elem_off, dense_off;  // dense_off: caller layout [cell][nu]
  long ndense = 0, nseg = 0;
  double* d_stage = nullptr;
  double* d_umax = nullptr;
  cudaGraphExec_t graph = nullptr;
  int graph_cur = -1, graph_launches = 0;
  int64_t launches = 0;
  // FP32 segment kernel: shape (faces per CTA, threads, persistent grid)
  // and its launch; segment tables are rebuilt when the shape changes
  int seg = 16, seg_t = 128, persist = 0;
  const void* seg_fn = nullptr;
  int seg_smem = 0, seg_grid = 0;
  int* d_segb = nullptr;
  int* d_segi0 = nullptr;
  int* d_segfirst = nullptr;
  int* d_nseg = nullptr;
  long seg_cap = 0;  // capacity of the segment tables (segments of 7 cells)
  // pool form (kb_pool_*): instance slots that requests join and leave, and
  // first-fit allocators of the cell, element and velocity ranges
  bool pool = false;
  std::vector<char> used;
  std::map<long, long> free_cells, free_elems, free_vels;  // offset -> length
};

static int bfail(int code, const std::string& m) {
  kb::set_error(m);
  return code;
}

static int balloc(kb_batch* B, void** p, size_t bytes) {
  if (bytes == 0) bytes = 16;
  if (cudaMalloc(p, bytes) != cudaSuccess) {
    cudaGetLastError();
    return bfail(KB_ERR_NOMEM, "cudaMalloc failed (" + std::to_string(bytes) + " bytes)");
  }
  B->allocs.push_back(*p);
  return KB_OK;
}

extern "C" int kb_batch_destroy(kb_batch_t* B) {
  if (!B) return KB_OK;
  if (B->stream) cudaStreamSynchronize(B->stream);
  if (B->graph) cudaGraphExecDestroy(B->graph);
  for (void* p : B->allocs) cudaFree(p);
  if (B->stream) cudaStreamDestroy(B->stream);
  delete B;
  return KB_OK;
}

// Compiled shapes of the FP32 segment kernel (kb_batch_seg_a.cu, _b.cu).
const std::vector<kb::SegVariant>& kb::seg_variants() {
  static const std::vector<kb::SegVariant> v = [] {
    std::vector<kb::SegVariant> out;
    kb::seg_variants_a(out);
    kb::seg_variants_b(out);
    return out;
  }();
  return v;
}

// Segment tables for `seg` cells per segment (an instance's segments are
// consecutive).  Waits for the stream; invalidates the step graph.
static int batch_tables(kb_batch* B, int seg) {
  std::vector<int> seg_b, seg_i0, seg_first(B->n), nseg(B->n);
  std::vector<kb::SegDesc> seg_d;
  for (int b = 0; b < B->n; ++b) {
    seg_first[b] = (int)seg_b.size();
    nseg[b] = B->pool && !B->used[b] ? 0 : (B->nx[b] + seg - 1) / seg;
    for (int k = 0; k < nseg[b]; ++k) {
      seg_b.push_back(b);
      seg_i0.push_back(k * seg);
      if (B->prec == KB_PREC_FP32)
        seg_d.push_back({b, k * seg, B->nx[b], B->ng[b], B->nu[b], B->nus[b], (int)B->vel_off_h[b], 0,
                         B->cell_off[b], B->elem_off[b], 1.0 / B->dx[b], float(1.e-7 * B->dx[b]),
                         2.f * float(B->mu[b])});
    }
  }
  if ((long)seg_b.size() > B->seg_cap) return bfail(KB_ERR_ARG, "batch shape: segment table overflow");
  cudaStreamSynchronize(B->stream);
  bool ok = true;
  ok &= cudaMemcpy(B->d_segb, seg_b.data(), sizeof(int) * seg_b.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(B->d_segi0, seg_i0.data(), sizeof(int) * seg_i0.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy((void*)B->d.seg_d, seg_d.data(), sizeof(kb::SegDesc) * seg_d.size(), cudaMemcpyHostToDevice) ==
        cudaSuccess;
  ok &= cudaMemcpy(B->d_segfirst, seg_first.data(), sizeof(int) * B->n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(B->d_nseg, nseg.data(), sizeof(int) * B->n, cudaMemcpyHostToDevice) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    return bfail(KB_ERR_CUDA, "batch shape: segment table upload failed");
  }
  B->nseg = (long)seg_b.size();
  B->d.nseg_all = (int)B->nseg;
  B->seg = seg;
  if (B->graph) {
    cudaGraphExecDestroy(B->graph);
    B->graph = nullptr;
  }
  return KB_OK;
}

// Select the FP32 segment kernel's shape: its segment tables, the kernel's
// shared-memory limit, and the grid -- one CTA per segment, or (persist) as
// many CTAs as fit on the GPU at once, each looping over segments.  Runs
// outside any stream capture.
static int batch_set_shape(kb_batch* B, int seg, int threads, int persist) {
  const kb::SegVariant* var = nullptr;
  for (const auto& v : kb::seg_variants())
    if (v.seg == seg && v.threads == threads) var = &v;
  if (!var) return bfail(KB_ERR_ARG, "batch shape: no segment kernel for " + std::to_string(seg) +
                                         " cells x " + std::to_string(threads) + " threads");
  int rc = batch_tables(B, var->cells);
  if (rc != KB_OK) return rc;
  bool ok = true;
  const int smem = var->smem(B->d.sst_max, B->d.nu4_max);
  ok &= cudaFuncSetAttribute(var->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, var->smem_max) ==
        cudaSuccess;
  // the carveout of every step kernel (kb::prefer_max_shared): a pool that
  // shares the GPU with other solves' streams keeps their CTAs on common SMs
  kb::prefer_max_shared(var->fn);
  kb::prefer_max_shared((const void*)kb::k_batch_seg_res);
  int per = 0, dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  ok &= cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, var->fn, threads, smem) == cudaSuccess;
  if (!ok || per < 1) {
    cudaGetLastError();
    return bfail(KB_ERR_CUDA, "batch shape: kernel attributes refused");
  }
  B->seg = seg;
  B->seg_t = threads;
  B->persist = persist ? 1 : 0;
  B->seg_fn = var->fn;
  B->seg_smem = smem;
  B->seg_grid = persist ? (int)std::min<long>(B->nseg, (long)sms * per) : (int)B->nseg;
  if (B->pool && persist) B->seg_grid = sms * per;  // fixed, whatever the membership
  return KB_OK;
}

extern "C" int kb_batch_create(const kb_config_t* base, int32_t n, const int32_t* nx,
                               const int32_t* ngx, const int32_t* nu, const double* x0,
                               const double* x1, const double* umax, const double* mu_ref,
                               const double* u_all, const double* w_all, kb_batch_t** out) {
  if (!base || n <= 0 || !nx || !ngx || !nu || !x0 || !x1 || !umax || !mu_ref || !u_all ||
      !w_all || !out)
    return bfail(KB_ERR_ARG, "kb_batch_create: null argument or empty batch");
  if (base->dim != 1 || base->nf == 1) return bfail(KB_ERR_CONFIG, "batched solves are 1D2F1V");
  if (base->flux != KB_FLUX_KFVS) return bfail(KB_ERR_CONFIG, "batched solves use KFVS");
  if (base->bc[0] != KB_BC_FIX || base->bc[1] != KB_BC_FIX)
    return bfail(KB_ERR_CONFIG, "batched solves use fixed boundaries");
  if (base->interp_order != 2) return bfail(KB_ERR_CONFIG, "batched solves use van Leer slopes");
  if (base->precision != KB_PREC_FP64 && base->precision != KB_PREC_FP32)
    return bfail(KB_ERR_CONFIG, "unknown precision");
  for (int b = 0; b < n; ++b) {
    if (nx[b] < 3 || nu[b] < 1 || nu[b] > 256 || ngx[b] < 0 || ngx[b] > 2 || !(x1[b] > x0[b]))
      return bfail(KB_ERR_CONFIG, "instance " + std::to_string(b) +
                                      ": need nx >= 3, 1 <= nu <= 256, 0 <= ng <= 2, x1 > x0");
  }
  kb_batch* B = new kb_batch();
  B->prec = base->precision;
  B->n = n;
  B->nx.assign(nx, nx + n);
  B->ng.assign(ngx, ngx + n);
  B->nu.assign(nu, nu + n);
  std::vector<int> vel_off(n);
  std::vector<double> dx(n), rdx(n), dt(n, 0.0), mu(mu_ref, mu_ref + n), rmu(n);
  B->cell_off.resize(n);
  B->elem_off.resize(n);
  long cells = 0, elems = 0, vels = 0;
  B->nus.resize(n);
  B->dense_off.resize(n);
  long dense = 0;
  long seg_cap = 0;
  for (int b = 0; b < n; ++b) {
    B->cell_off[b] = cells;
    B->elem_off[b] = elems;
    B->dense_off[b] = dense;
    vel_off[b] = (int)vels;
    long nxt = nx[b] + 2 * ngx[b];
    B->nus[b] = (nu[b] + 3) / 4 * 4;
    cells += nxt;
    elems += nxt * B->nus[b];
    dense += nxt * nu[b];
    vels += nu[b];
    dx[b] = (x1[b] - x0[b]) / nx[b];
    rdx[b] = 1.0 / dx[b];
    rmu[b] = 1.0 / (2.0 * mu[b]);
    seg_cap += (nx[b] + 6) / 7 + 1;  // the shortest segment length the tuner offers (a pool's members: one more)
  }
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int seg64 = kb::seg64_cells(cells, sms);
  if (B->prec == KB_PREC_FP64) {
    seg_cap = 0;
    for (int b = 0; b < n; ++b) seg_cap += (nx[b] + seg64 - 1) / seg64;
  }
  B->dx = dx;
  B->mu = mu;
  B->vel_off_h.assign(vel_off.begin(), vel_off.end());
  B->ndense = dense;
  B->seg_cap = seg_cap;
  B->ncell = cells;
  B->nelem = elems;
  B->nvel = vels;
  auto fail_out = [&](int rc) {
    kb_batch_destroy(B);
    return rc;
  };
  if (cudaStreamCreateWithFlags(&B->stream, cudaStreamNonBlocking) != cudaSuccess)
    return fail_out(bfail(KB_ERR_CUDA, "cudaStreamCreate failed"));
  void* p;
  int rc;
#define BALLOC(dst, T, count)                                              \
  if ((rc = balloc(B, &p, sizeof(T) * (size_t)(count))) != KB_OK) return fail_out(rc); \
  dst = (T*)p;
  int *d_nx, *d_ng, *d_nu, *d_vo, *d_active, *d_status;
  int *d_nus, *d_segb, *d_segi0, *d_segfirst, *d_nseg;
  double* d_respart;
  long *d_co, *d_eo;
  double *d_dx, *d_rdx, *d_dt, *d_rmu, *d_mc64, *d_u, *d_w, *d_wv, *d_prim, *d_res;
  float *d_uf, *d_wf, *d_ul, *d_mc;
  BALLOC(d_nx, int, n);
  BALLOC(d_ng, int, n);
  BALLOC(d_nu, int, n);
  BALLOC(d_nus, int, n);
  BALLOC(d_segb, int, B->seg_cap);
  BALLOC(d_segi0, int, B->seg_cap);
  BALLOC(B->d.seg_d, const kb::SegDesc, B->prec == KB_PREC_FP32 ? B->seg_cap : 0);
  BALLOC(d_segfirst, int, n);
  BALLOC(d_nseg, int, n);
  BALLOC(d_respart, double, B->seg_cap * 8);
  BALLOC(d_vo, int, n);
  BALLOC(d_active, int, n);
  BALLOC(d_status, int, 1);
  BALLOC(d_co, long, n);
  BALLOC(d_eo, long, n);
  BALLOC(d_dx, double, n);
  BALLOC(d_dt, double, n);
  BALLOC(d_rdx, double, n);
  BALLOC(d_rmu, double, n);
  BALLOC(d_u, double, vels);
  BALLOC(d_wv, double, vels);
  BALLOC(d_uf, float, vels);
  BALLOC(d_ul, float, vels);
  BALLOC(d_wf, float, vels);
  BALLOC(d_w, double, cells * 4);
  BALLOC(d_prim, double, cells * 4);
  BALLOC(d_mc, float, B->prec == KB_PREC_FP32 ? cells * 8 : 0);
  BALLOC(d_mc64, double, B->prec == KB_PREC_FP64 ? cells * 4 : 0);
  BALLOC(d_res, double, (size_t)n * 4);
  BALLOC(B->d_umax, double, n);
  size_t esz = B->prec == KB_PREC_FP64 ? 8 : 4;
  for (int k = 0; k < 2; ++k) {
    if ((rc = balloc(B, &B->h[k], esz * elems)) != KB_OK) return fail_out(rc);
    if ((rc = balloc(B, &B->bq[k], esz * elems)) != KB_OK) return fail_out(rc);
  }
  BALLOC(B->d_stage, double, elems);
  // padding values of the distribution rows stay zero in both buffers
  for (int k = 0; k < 2; ++k) {
    cudaMemset(B->h[k], 0, esz * elems);
    cudaMemset(B->bq[k], 0, esz * elems);
  }
#undef BALLOC
  std::vector<float> uf(u_all, u_all + vels), wf(w_all, w_all + vels), ul(vels);
  for (long k = 0; k < vels; ++k) ul[k] = float(u_all[k] - (double)uf[k]);
  std::vector<int> ones(n, 1);
  bool ok = true;
  ok &= cudaMemcpy(d_nx, nx, sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_ng, ngx, sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_nu, nu, sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_nus, B->nus.data(), sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemset(d_respart, 0, sizeof(double) * B->seg_cap * 8) == cudaSuccess;
  ok &= cudaMemcpy(d_vo, vel_off.data(), sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_active, ones.data(), sizeof(int) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_co, B->cell_off.data(), sizeof(long) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_eo, B->elem_off.data(), sizeof(long) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_dx, dx.data(), sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_dt, dt.data(), sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_rdx, rdx.data(), sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_rmu, rmu.data(), sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_u, u_all, sizeof(double) * vels, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_wv, w_all, sizeof(double) * vels, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_uf, uf.data(), sizeof(float) * vels, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_ul, ul.data(), sizeof(float) * vels, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(d_wf, wf.data(), sizeof(float) * vels, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(B->d_umax, umax, sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemset(d_status, 0, sizeof(int)) == cudaSuccess;
  ok &= cudaMemset(d_res, 0, sizeof(double) * n * 4) == cudaSuccess;
  if (!ok) return fail_out(bfail(KB_ERR_CUDA, "batch table upload failed"));
  kb::BatchDev& d = B->d;
  d.n = n;
  d.nx = d_nx;
  d.ng = d_ng;
  d.nu = d_nu;
  d.nus = d_nus;
  d.seg_b = d_segb;
  d.seg_i0 = d_segi0;
  d.seg_first = d_segfirst;
  d.nseg = d_nseg;
  B->d_segb = d_segb;
  B->d_segi0 = d_segi0;
  B->d_segfirst = d_segfirst;
  B->d_nseg = d_nseg;
  d.respart = d_respart;
  d.sst_max = 4;
  d.nu4_max = 4;
  for (int b = 0; b < n; ++b) {
    d.sst_max = std::max(d.sst_max, kb::seg_stride(B->nus[b]));
    d.nu4_max = std::max(d.nu4_max, B->nus[b]);
  }
  d.cell_off = d_co;
  d.elem_off = d_eo;
  d.vel_off = d_vo;
  d.dx = d_dx;
  d.dt = d_dt;
  d.rdx = d_rdx;
  d.rmu = d_rmu;
  d.u = d_u;
  d.wt = d_wv;
  d.uf = d_uf;
  d.ul = d_ul;
  d.wtf = d_wf;
  d.w = d_w;
  d.prim = d_prim;
  d.mc = d_mc;
  d.mc64 = d_mc64;
  d.residual = d_res;
  d.active = d_active;
  d.status = d_status;
  d.K = base->K;
  d.gamma = base->gamma;
  d.omega = base->omega;
  d.Pr = base->Pr;
  kb::seg_gas(d);
  d.tol = 0.0;
  d.coll = base->collision;
  d.clock = nullptr;
  d.fw = nullptr;
  if (B->prec == KB_PREC_FP64) {
    if (!kb::seg64_prepare()) return fail_out(bfail(KB_ERR_CUDA, "FP64 segment kernel attributes refused"));
    if ((rc = batch_tables(B, seg64)) != KB_OK) return fail_out(rc);
  }
  if (B->prec == KB_PREC_FP32 && (rc = batch_set_shape(B, 16, 128, 0)) != KB_OK)
    return fail_out(rc);
  *out = B;
  return KB_OK;
}

extern "C" int kb_batch_upload(kb_batch_t* B, const double* w, const double* prim,
                               const double* h, const double* bq) {
  if (B && B->pool) return bfail(KB_ERR_STATE, "pools move state per slot (kb_pool_add / kb_pool_download)");
  if (!B || !w || !prim || !h || !bq) return bfail(KB_ERR_ARG, "kb_batch_upload: null argument");
  std::vector<double> w4(B->ncell * 4, 0.0), p4(B->ncell * 4, 0.0);
  for (long c = 0; c < B->ncell; ++c)
    for (int k = 0; k < 3; ++k) {
      w4[c * 4 + k] = w[c * 3 + k];
      p4[c * 4 + k] = prim[c * 3 + k];
    }
  if (cudaMemcpy(B->d.w, w4.data(), sizeof(double) * w4.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(B->d.prim, p4.data(), sizeof(double) * p4.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return bfail(KB_ERR_CUDA, "kb_batch_upload: copy failed");
  const long n = B->nelem;
  const unsigned g = (unsigned)((n + 255) / 256);
  std::vector<double> pad(n, 0.0);  // caller rows of nu values -> padded rows
  for (int which = 0; which < 2; ++which) {
    const double* src = which == 0 ? h : bq;
    for (int b = 0; b < B->n; ++b) {
      const long nxt = B->nx[b] + 2 * B->ng[b];
      for (long c = 0; c < nxt; ++c)
        std::memcpy(&pad[B->elem_off[b] + c * B->nus[b]], src + B->dense_off[b] + c * B->nu[b],
                    sizeof(double) * B->nu[b]);
    }
    if (cudaMemcpy(B->d_stage, pad.data(), sizeof(double) * n, cudaMemcpyHostToDevice) != cudaSuccess)
      return bfail(KB_ERR_CUDA, "kb_batch_upload: copy failed");
    for (int k = 0; k < 2; ++k) {
      void* dst = which == 0 ? B->h[k] : B->bq[k];
      if (B->prec == KB_PREC_FP64)
        kb::k_batch_convert<double><<<g, 256, 0, B->stream>>>((double*)dst, B->d_stage, n);
      else
        kb::k_batch_convert<float><<<g, 256, 0, B->stream>>>((float*)dst, B->d_stage, n);
      B->launches++;
    }
    cudaStreamSynchronize(B->stream);
  }
  {  // the step reads each cell's Maxwellian coefficients
    int maxc = 1;
    for (int b = 0; b < B->n; ++b) maxc = std::max(maxc, B->nx[b] + 2 * B->ng[b]);
    if (B->prec == KB_PREC_FP32) kb::seg_mcache_launch(B->d, B->n, maxc, B->stream);
    else kb::seg64_mcache_launch(B->d, B->n, maxc, B->stream);
    B->launches++;
    cudaStreamSynchronize(B->stream);
  }
  std::vector<int> ones(B->n, 1);
  cudaMemcpy((void*)B->d.active, ones.data(), sizeof(int) * B->n, cudaMemcpyHostToDevice);
  cudaMemset(B->d.status, 0, sizeof(int));
  B->cur = 0;
  if (cudaGetLastError() != cudaSuccess) return bfail(KB_ERR_CUDA, "kb_batch_upload failed");
  return KB_OK;
}

extern "C" int kb_batch_init_equilibrium(kb_batch_t* B, const double* w, const double* prim) {
  if (B && B->pool) return bfail(KB_ERR_STATE, "pools move state per slot (kb_pool_add / kb_pool_download)");
  if (!B || !w || !prim) return bfail(KB_ERR_ARG, "kb_batch_init_equilibrium: null argument");
  std::vector<double> w4(B->ncell * 4, 0.0), p4(B->ncell * 4, 0.0);
  for (long c = 0; c < B->ncell; ++c)
    for (int k = 0; k < 3; ++k) {
      w4[c * 4 + k] = w[c * 3 + k];
      p4[c * 4 + k] = prim[c * 3 + k];
    }
  if (cudaMemcpy(B->d.w, w4.data(), sizeof(double) * w4.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(B->d.prim, p4.data(), sizeof(double) * p4.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return bfail(KB_ERR_CUDA, "kb_batch_init_equilibrium: copy failed");
  int maxc = 1;
  for (int b = 0; b < B->n; ++b) maxc = std::max(maxc, B->nx[b] + 2 * B->ng[b]);
  const dim3 grid((unsigned)maxc, (unsigned)B->n);
  if (B->prec == KB_PREC_FP64) {
    kb::k_batch_init_eq64<<<grid, 128, 0, B->stream>>>(B->d, (double*)B->h[0], (double*)B->bq[0],
                                                       (double*)B->h[1], (double*)B->bq[1]);
    kb::seg64_mcache_launch(B->d, B->n, maxc, B->stream);
    B->launches++;
  } else {
    // (the FP64 work of a cell's coefficients by one thread per cell: every
    // warp of the cell's own CTA doing it took 476 us for 115,000 cells)
    kb::seg_mcache_launch(B->d, B->n, maxc, B->stream);
    kb::k_batch_init_eq32<<<grid, 128, 0, B->stream>>>(B->d, 0, (float*)B->h[0], (float*)B->bq[0],
                                                       (float*)B->h[1], (float*)B->bq[1]);
    B->launches++;
  }
  B->launches++;
  std::vector<int> ones(B->n, 1);
  cudaMemcpyAsync((void*)B->d.active, ones.data(), sizeof(int) * B->n, cudaMemcpyHostToDevice, B->stream);
  cudaMemsetAsync(B->d.status, 0, sizeof(int), B->stream);
  if (cudaStreamSynchronize(B->stream) != cudaSuccess)
    return bfail(KB_ERR_CUDA, std::string("kb_batch_init_equilibrium: ") +
                                  cudaGetErrorString(cudaGetLastError()));
  B->cur = 0;
  return KB_OK;
}

extern "C" int kb_batch_download(kb_batch_t* B, double* w, double* prim, double* h, double* bq) {
  if (B && B->pool) return bfail(KB_ERR_STATE, "pools move state per slot (kb_pool_add / kb_pool_download)");
  if (!B) return bfail(KB_ERR_ARG, "kb_batch_download: null handle");
  cudaStreamSynchronize(B->stream);
  if (w || prim) {
    std::vector<double> w4(B->ncell * 4), p4(B->ncell * 4);
    cudaMemcpy(w4.data(), B->d.w, sizeof(double) * w4.size(), cudaMemcpyDeviceToHost);
    cudaMemcpy(p4.data(), B->d.prim, sizeof(double) * p4.size(), cudaMemcpyDeviceToHost);
    for (long c = 0; c < B->ncell; ++c)
      for (int k = 0; k < 3; ++k) {
        if (w) w[c * 3 + k] = w4[c * 4 + k];
        if (prim) prim[c * 3 + k] = p4[c * 4 + k];
      }
  }
  const long n = B->nelem;
  const unsigned g = (unsigned)((n + 255) / 256);
  std::vector<double> pad(n);
  for (int which = 0; which < 2; ++which) {
    double* dst = which == 0 ? h : bq;
    if (!dst) continue;
    const void* src = which == 0 ? B->h[B->cur] : B->bq[B->cur];
    if (B->prec == KB_PREC_FP64)
      kb::k_batch_back<double><<<g, 256, 0, B->stream>>>(B->d_stage, (const double*)src, n);
    else
      kb::k_batch_back<float><<<g, 256, 0, B->stream>>>(B->d_stage, (const float*)src, n);
    B->launches++;
    cudaStreamSynchronize(B->stream);
    cudaMemcpy(pad.data(), B->d_stage, sizeof(double) * n, cudaMemcpyDeviceToHost);
    for (int b = 0; b < B->n; ++b) {
      const long nxt = B->nx[b] + 2 * B->ng[b];
      for (long c = 0; c < nxt; ++c)
        std::memcpy(dst + B->dense_off[b] + c * B->nu[b], &pad[B->elem_off[b] + c * B->nus[b]],
                    sizeof(double) * B->nu[b]);
    }
  }
  if (cudaGetLastError() != cudaSuccess) return bfail(KB_ERR_CUDA, "kb_batch_download failed");
  return KB_OK;
}

extern "C" int kb_batch_timestep(kb_batch_t* B, double cfl, double* dt_out) {
  if (B && B->pool) return bfail(KB_ERR_STATE, "pool time steps are set per slot by kb_pool_add");
  if (!B) return bfail(KB_ERR_ARG, "kb_batch_timestep: null handle");
  kb::k_batch_timestep<<<B->n, 256, 0, B->stream>>>(B->d, B->d_umax, cfl, (double*)B->d.dt);
  B->launches++;
  cudaStreamSynchronize(B->stream);
  if (dt_out) cudaMemcpy(dt_out, B->d.dt, sizeof(double) * B->n, cudaMemcpyDeviceToHost);
  if (cudaGetLastError() != cudaSuccess) return bfail(KB_ERR_CUDA, "kb_batch_timestep failed");
  return KB_OK;
}

extern "C" int kb_batch_set_dt(kb_batch_t* B, const double* dt) {
  if (B && B->pool) return bfail(KB_ERR_STATE, "pool time steps are set per slot by kb_pool_add");
  if (!B || !dt) return bfail(KB_ERR_ARG, "kb_batch_set_dt: null argument");
  if (cudaMemcpy((void*)B->d.dt, dt, sizeof(double) * B->n, cudaMemcpyHostToDevice) != cudaSuccess)
    return bfail(KB_ERR_CUDA, "kb_batch_set_dt failed");
  return KB_OK;
}

// One step from buffer `cur`.  The residual kernel sets residuals and
// convergence flags; with tol = 0 no flag can change, so only the last step of
// a call needs it (res).  Returns the kernels launched, or KB_ERR_CUDA when a
// launch was refused (seen nowhere else).
static int batch_launch(kb_batch* B, int cur, bool res) {
  int n = 0;
  if (B->prec == KB_PREC_FP32) {  // fused segments (one pass over HBM)
    const float* hin = (const float*)B->h[cur];
    const float* bin = (const float*)B->bq[cur];
    float* hout = (float*)B->h[cur ^ 1];
    float* bout = (float*)B->bq[cur ^ 1];
    int slot = -1, want = res;
    void* args[] = {(void*)&B->d, (void*)&hin, (void*)&bin, (void*)&hout, (void*)&bout, (void*)&slot, (void*)&want};
    if (B->seg_grid > 0) {  // an empty pool has no segments
      kb::launch_after(B->seg_fn, dim3((unsigned)B->seg_grid), dim3((unsigned)B->seg_t),
                       (size_t)B->seg_smem, B->stream, args);
      ++n;
    }
  } else {
    kb::seg64_launch(B->d, B->seg, (const double*)B->h[cur], (const double*)B->bq[cur],
                     (double*)B->h[cur ^ 1], (double*)B->bq[cur ^ 1], res, -1, B->stream);
    ++n;
  }
  if (res) {
    kb::seg_res_launch(B->d, B->stream);
    ++n;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return bfail(KB_ERR_CUDA, std::string("batch step launch: ") + cudaGetErrorString(e));
  return n;
}

// Two steps (ping and pong) captured once as a CUDA graph and replayed.
static int batch_graph(kb_batch* B) {
  if (B->graph && B->graph_cur == B->cur) return KB_OK;
  if (B->graph) {
    cudaGraphExecDestroy(B->graph);
    B->graph = nullptr;
  }
  cudaGraph_t g;
  if (cudaStreamBeginCapture(B->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
    return bfail(KB_ERR_CUDA, "graph capture failed to start");
  const bool res = B->d.tol > 0.0;  // flags may change at every step
  const int n0 = batch_launch(B, B->cur, res), n1 = n0 < 0 ? n0 : batch_launch(B, B->cur ^ 1, res);
  const cudaError_t ec = cudaStreamEndCapture(B->stream, &g);
  cudaGetLastError();  // (a refused launch ends the capture too; the next call starts clean)
  if (n1 < 0) {
    if (ec == cudaSuccess) cudaGraphDestroy(g);
    return n1;
  }
  if (ec != cudaSuccess) return bfail(KB_ERR_CUDA, "graph capture failed");
  B->graph_launches = n0 + n1;
  cudaError_t e = cudaGraphInstantiate(&B->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return bfail(KB_ERR_CUDA, "graph instantiation failed");
  B->graph_cur = B->cur;
  return KB_OK;
}

extern "C" int kb_batch_step(kb_batch_t* B, int32_t nsteps, double tol, double* residual,
                             int32_t* active) {
  if (!B) return bfail(KB_ERR_ARG, "kb_batch_step: null handle");
  if (nsteps < 0) return bfail(KB_ERR_ARG, "kb_batch_step: nsteps must be >= 0");
  if (B->d.tol != tol) {
    B->d.tol = tol;
    if (B->graph) {
      cudaGraphExecDestroy(B->graph);
      B->graph = nullptr;
    }
  }
  // pairs of steps replayed, the last one or two launched with the residual
  int left = nsteps;
  if (left > 2) {
    int rc = batch_graph(B);
    if (rc != KB_OK) return rc;
    for (; left > 2; left -= 2) {
      if (cudaGraphLaunch(B->graph, B->stream) != cudaSuccess)
        return bfail(KB_ERR_CUDA, "graph launch failed");
      B->launches += B->graph_launches;
    }
  }
  for (; left > 0; --left) {
    const int k = batch_launch(B, B->cur, left == 1 || tol > 0.0);
    if (k < 0) return k;
    B->launches += k;
    B->cur ^= 1;
  }
  if (cudaStreamSynchronize(B->stream) != cudaSuccess)
    return bfail(KB_ERR_CUDA, std::string("batch step failed: ") + cudaGetErrorString(cudaGetLastError()));
  if (residual)
    cudaMemcpy(residual, B->d.residual, sizeof(double) * 4 * B->n, cudaMemcpyDeviceToHost);
  if (active) cudaMemcpy(active, B->d.active, sizeof(int) * B->n, cudaMemcpyDeviceToHost);
  int st = 0;
  cudaMemcpy(&st, B->d.status, sizeof(int), cudaMemcpyDeviceToHost);
  if (st) return bfail(KB_ERR_NUMERIC, "non-finite or non-positive density / lambda in a batched solve");
  return KB_OK;
}

extern "C" int kb_batch_set_tuning(kb_batch_t* B, const int32_t* params, int32_t n) {
  if (!B || !params || n < 1) return bfail(KB_ERR_ARG, "kb_batch_set_tuning: null argument");
  if (B->prec != KB_PREC_FP32) return KB_OK;  // the FP64 form has one shape
  const int seg = params[0] > 0 ? params[0] : 16;
  const int thr = n > 1 && params[1] > 0 ? params[1] : 128;
  const int per = n > 2 ? params[2] : 0;
  return batch_set_shape(B, seg, thr, per);
}

extern "C" int kb_batch_get_tuning(kb_batch_t* B, int32_t* params, int32_t n) {
  if (!B || !params) return bfail(KB_ERR_ARG, "kb_batch_get_tuning: null argument");
  const int32_t v[3] = {B->seg, B->seg_t, B->persist};
  for (int k = 0; k < n && k < 3; ++k) params[k] = v[k];
  return KB_OK;
}

extern "C" int kb_batch_info(kb_batch_t* B, int64_t* elems, int64_t* launches) {
  if (!B) return bfail(KB_ERR_ARG, "kb_batch_info: null handle");
  if (elems) *elems = B->nelem;
  if (launches) *launches = B->launches;
  return KB_OK;
}

// ----------------------------------------------------------------- pool
// Continuous batching of 1D2F1V solves: a pool of instance slots with
// capacity fixed at creation; a request joins between steps (kb_pool_add
// places it in free cell / element / velocity ranges, builds its equilibrium
// state on the device and computes its time step) and leaves between steps
// (kb_pool_remove frees its ranges); kb_batch_step advances every resident
// instance with the same fused launch per step.  Only the segment tables and
// the per-slot scalars change on a join or leave (small host-to-device
// copies); the step graph is re-captured at the next step.

static long range_alloc(std::map<long, long>& fr, long n) {
  for (auto it = fr.begin(); it != fr.end(); ++it) {
    if (it->second >= n) {
      const long off = it->first, len = it->second;
      fr.erase(it);
      if (len > n) fr[off + n] = len - n;
      return off;
    }
  }
  return -1;
}

static void range_free(std::map<long, long>& fr, long off, long n) {
  auto it = fr.emplace(off, n).first;
  auto nx = std::next(it);
  if (nx != fr.end() && it->first + it->second == nx->first) {
    it->second += nx->second;
    fr.erase(nx);
  }
  if (it != fr.begin()) {
    auto pv = std::prev(it);
    if (pv->first + pv->second == it->first) {
      pv->second += it->second;
      fr.erase(it);
    }
  }
}

extern "C" int kb_pool_create(const kb_config_t* base, int32_t max_instances, int64_t max_cells,
                              int32_t max_nu, kb_batch_t** out) {
  if (!base || !out || max_instances < 1 || max_cells < 3 * (int64_t)max_instances || max_nu < 1)
    return bfail(KB_ERR_ARG, "kb_pool_create: null argument or empty capacity");
  if (base->dim != 1 || base->nf == 1) return bfail(KB_ERR_CONFIG, "pooled solves are 1D2F1V");
  if (base->precision != KB_PREC_FP32) return bfail(KB_ERR_CONFIG, "pooled solves use the FP32 split form");
  if (base->flux != KB_FLUX_KFVS) return bfail(KB_ERR_CONFIG, "pooled solves use KFVS");
  if (base->bc[0] != KB_BC_FIX || base->bc[1] != KB_BC_FIX)
    return bfail(KB_ERR_CONFIG, "pooled solves use fixed boundaries");
  if (max_nu > kb::SEG_MAXNU) return bfail(KB_ERR_CONFIG, "pooled solves have at most 256 velocities");
  // placeholder instances of max_nu velocities and max_cells cells in all
  // size the arrays (cells x max_nu distribution values, n x max_nu
  // velocities); their slots are then released
  const int n = max_instances;
  std::vector<int32_t> nx(n, 3), ng(n, 0), nu(n, max_nu);
  nx[0] = (int32_t)(max_cells - 3 * (int64_t)(n - 1));
  std::vector<double> x0(n, 0.0), x1(n, 1.0), um(n, 1.0), mu(n, base->mu_ref);
  std::vector<double> uu((size_t)n * max_nu, 0.0), ww((size_t)n * max_nu, 1.0);
  kb_config_t c = *base;
  c.nu = max_nu;
  kb_batch_t* B = nullptr;
  int rc = kb_batch_create(&c, n, nx.data(), ng.data(), nu.data(), x0.data(), x1.data(),
                           um.data(), mu.data(), uu.data(), ww.data(), &B);
  if (rc != KB_OK) return rc;
  B->pool = true;
  B->used.assign(n, 0);
  B->free_cells[0] = B->ncell;
  B->free_elems[0] = B->nelem;
  B->free_vels[0] = B->nvel;
  B->vel_off_h.assign(n, 0);
  std::vector<int> zeros(n, 0);
  cudaMemcpy((void*)B->d.active, zeros.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
  for (int b = 0; b < n; ++b) B->nx[b] = 0;
  rc = batch_set_shape(B, 16, 128, 1);
  if (rc != KB_OK) {
    kb_batch_destroy(B);
    return rc;
  }
  *out = B;
  return KB_OK;
}

template <typename T>
static bool put1(const T* dev, int b, T v) {
  return cudaMemcpy((void*)(dev + b), &v, sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
}

extern "C" int kb_pool_add(kb_batch_t* B, int32_t nx, int32_t ngx, int32_t nu, double x0, double x1,
                           double umax, double mu_ref, const double* u, const double* wts,
                           const double* w, const double* prim, double cfl, int32_t* slot,
                           double* dt_out) {
  if (!B || !B->pool || !u || !wts || !w || !prim || !slot) return bfail(KB_ERR_ARG, "kb_pool_add: null argument");
  if (nx < 3 || ngx < 0 || ngx > 2 || nu < 1 || nu > (int)B->d.nu4_max || !(x1 > x0) || !(cfl > 0.0))
    return bfail(KB_ERR_CONFIG, "kb_pool_add: invalid instance");
  int b = -1;
  for (int k = 0; k < B->n && b < 0; ++k)
    if (!B->used[k]) b = k;
  if (b < 0) return bfail(KB_ERR_NOMEM, "kb_pool_add: no free slot");
  const long nxt = nx + 2 * ngx, nus = (nu + 3) / 4 * 4;
  const long co = range_alloc(B->free_cells, nxt);
  const long eo = co < 0 ? -1 : range_alloc(B->free_elems, nxt * nus);
  const long vo = eo < 0 ? -1 : range_alloc(B->free_vels, nu);
  if (vo < 0) {
    if (eo >= 0) range_free(B->free_elems, eo, nxt * nus);
    if (co >= 0) range_free(B->free_cells, co, nxt);
    return bfail(KB_ERR_NOMEM, "kb_pool_add: the pool's cell or velocity capacity is used up");
  }
  cudaStreamSynchronize(B->stream);
  B->used[b] = 1;
  B->nx[b] = nx;
  B->ng[b] = ngx;
  B->nu[b] = nu;
  B->nus[b] = (int)nus;
  B->cell_off[b] = co;
  B->elem_off[b] = eo;
  B->vel_off_h[b] = vo;
  const double dx = (x1 - x0) / nx;
  B->dx[b] = dx;
  B->mu[b] = mu_ref;
  bool ok = put1(B->d.nx, b, (int)nx) && put1(B->d.ng, b, (int)ngx) && put1(B->d.nu, b, (int)nu) &&
            put1(B->d.nus, b, (int)nus) && put1(B->d.cell_off, b, co) && put1(B->d.elem_off, b, eo) &&
            put1(B->d.vel_off, b, (int)vo) && put1(B->d.dx, b, dx) &&
            put1(B->d.rdx, b, 1.0 / dx) && put1(B->d.rmu, b, 1.0 / (2.0 * mu_ref)) &&
            put1((const double*)B->d_umax, b, umax);
  std::vector<float> uf(nu), ul(nu), wf(nu);
  for (int k = 0; k < nu; ++k) {
    uf[k] = float(u[k]);
    ul[k] = float(u[k] - (double)uf[k]);
    wf[k] = float(wts[k]);
  }
  ok &= cudaMemcpy((void*)(B->d.u + vo), u, sizeof(double) * nu, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy((void*)(B->d.wt + vo), wts, sizeof(double) * nu, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy((void*)(B->d.uf + vo), uf.data(), sizeof(float) * nu, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy((void*)(B->d.ul + vo), ul.data(), sizeof(float) * nu, cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy((void*)(B->d.wtf + vo), wf.data(), sizeof(float) * nu, cudaMemcpyHostToDevice) == cudaSuccess;
  std::vector<double> w4(nxt * 4, 0.0), p4(nxt * 4, 0.0);
  for (long c = 0; c < nxt; ++c)
    for (int k = 0; k < 3; ++k) {
      w4[c * 4 + k] = w[c * 3 + k];
      p4[c * 4 + k] = prim[c * 3 + k];
    }
  ok &= cudaMemcpy(B->d.w + co * 4, w4.data(), sizeof(double) * w4.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  ok &= cudaMemcpy(B->d.prim + co * 4, p4.data(), sizeof(double) * p4.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  if (!ok) return bfail(KB_ERR_CUDA, "kb_pool_add: copy failed");
  kb::seg_mcache_launch(B->d, 1, (int)nxt, B->stream, b);
  const int cur = B->cur;  // the buffer the next step reads: 1 after an odd number of steps
  kb::k_batch_init_eq32<<<dim3((unsigned)nxt, 1), 128, 0, B->stream>>>(
      B->d, b, (float*)B->h[cur], (float*)B->bq[cur], (float*)B->h[cur ^ 1], (float*)B->bq[cur ^ 1]);
  kb::k_batch_timestep<<<1, 256, 0, B->stream>>>(B->d, B->d_umax, cfl, (double*)B->d.dt, b);
  B->launches += 3;
  double dt = 0.0;
  ok &= cudaStreamSynchronize(B->stream) == cudaSuccess;
  ok &= cudaMemcpy(&dt, B->d.dt + b, sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess;
  ok &= put1((const int*)B->d.active, b, 1);
  const double zero4[4] = {0, 0, 0, 0};
  ok &= cudaMemcpy(B->d.residual + (long)b * 4, zero4, sizeof(zero4), cudaMemcpyHostToDevice) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    return bfail(KB_ERR_CUDA, "kb_pool_add: device set-up failed");
  }
  int rc = batch_set_shape(B, B->seg, B->seg_t, B->persist);
  if (rc != KB_OK) return rc;
  *slot = b;
  if (dt_out) *dt_out = dt;
  return KB_OK;
}

extern "C" int kb_pool_remove(kb_batch_t* B, int32_t slot) {
  if (!B || !B->pool || slot < 0 || slot >= B->n || !B->used[slot])
    return bfail(KB_ERR_ARG, "kb_pool_remove: no such slot");
  cudaStreamSynchronize(B->stream);
  const long nxt = B->nx[slot] + 2 * B->ng[slot];
  range_free(B->free_cells, B->cell_off[slot], nxt);
  range_free(B->free_elems, B->elem_off[slot], nxt * B->nus[slot]);
  range_free(B->free_vels, B->vel_off_h[slot], B->nu[slot]);
  B->used[slot] = 0;
  B->nx[slot] = 0;
  if (!put1((const int*)B->d.active, slot, 0)) return bfail(KB_ERR_CUDA, "kb_pool_remove: copy failed");
  return batch_set_shape(B, B->seg, B->seg_t, B->persist);
}

extern "C" int kb_pool_download(kb_batch_t* B, int32_t slot, double* w, double* prim, double* h,
                                double* bq) {
  if (!B || !B->pool || slot < 0 || slot >= B->n || !B->used[slot])
    return bfail(KB_ERR_ARG, "kb_pool_download: no such slot");
  cudaStreamSynchronize(B->stream);
  const long nxt = B->nx[slot] + 2 * B->ng[slot], co = B->cell_off[slot];
  const int nu = B->nu[slot], nus = B->nus[slot];
  bool ok = true;
  if (w || prim) {
    std::vector<double> a4(nxt * 4);
    for (int which = 0; which < 2; ++which) {
      double* dst = which == 0 ? w : prim;
      if (!dst) continue;
      ok &= cudaMemcpy(a4.data(), (which == 0 ? B->d.w : B->d.prim) + co * 4, sizeof(double) * a4.size(),
                       cudaMemcpyDeviceToHost) == cudaSuccess;
      for (long c = 0; c < nxt; ++c)
        for (int k = 0; k < 3; ++k) dst[c * 3 + k] = a4[c * 4 + k];
    }
  }
  const long ne = nxt * nus, eo = B->elem_off[slot];
  std::vector<double> stage(ne);
  for (int which = 0; which < 2; ++which) {
    double* dst = which == 0 ? h : bq;
    if (!dst) continue;
    const float* src = (const float*)(which == 0 ? B->h[B->cur] : B->bq[B->cur]) + eo;
    kb::k_batch_back<float><<<(unsigned)((ne + 255) / 256), 256, 0, B->stream>>>(B->d_stage, src, ne);
    B->launches++;
    ok &= cudaStreamSynchronize(B->stream) == cudaSuccess;
    ok &= cudaMemcpy(stage.data(), B->d_stage, sizeof(double) * ne, cudaMemcpyDeviceToHost) == cudaSuccess;
    for (long c = 0; c < nxt; ++c) std::memcpy(dst + c * nu, &stage[c * nus], sizeof(double) * nu);
  }
  if (!ok) return bfail(KB_ERR_CUDA, "kb_pool_download: copy failed");
  return KB_OK;
}
