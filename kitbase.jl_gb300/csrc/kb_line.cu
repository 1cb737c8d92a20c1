// kb_line.cu -- single 1D2F1V solves through the fused segment kernels.
//
// A 1D solve has a few tens of thousands of cell-velocity points: its step is
// bound by the latency of the kernels it is made of, not by their work.  The
// general form launches five (face parameters, face moments, cell parameters,
// update, residual), each a chain of global loads and FP64 divisions on a
// handful of CTAs; the segment kernels of the batch do the step in one launch,
// with the same layout of w, prim, h and b.
#include "kb_line.cuh"

#include <vector>

namespace kb {

bool line_covers(const kb_config_t& c) {
  return c.dim == 1 && c.nf != 1 && c.flux == KB_FLUX_KFVS && c.interp_order == 2 &&
         c.bc[0] == KB_BC_FIX && c.bc[1] == KB_BC_FIX && c.nu <= SEG_MAXNU;
}

static const SegVariant kShort = {4, 128, 3, (const void*)k_batch_seg<3, 128, true>, seg_smem<3, 128>,
                                  seg_smem_max<3, 128>()};
static const SegVariant kLong = {16, 128, 15, (const void*)k_batch_seg<15, 128, true>, seg_smem<15, 128>,
                                 seg_smem_max<15, 128>()};

// FP32: segments of three cells while the GPU holds all of them at once, and so a
// step is one segment's latency; longer lines, whose segments queue, by fifteen,
// which read 19 rows of the window for 15 cells and not 7 for 3, and run the
// cell phase a fifth as often.  us a step, 3 / 15 cells (the general form):
// 1000 x 100 7.2 / 9.2 (62), 2048 x 48 12.0 / 7.6 (59), 2048 x 256 15.5 / 13.5
// (73), 20,000 x 256 117 / 51 (159), 100,000 x 48 436 / 84 (412), 400,000 x 48
// 1,865 / 350 (1,551).
static const SegVariant* line_variant(const kb_config_t& c, int vstride, int sms) {
  for (const SegVariant* v : {&kShort, &kLong}) {
    if (cudaFuncSetAttribute(v->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v->smem_max) != cudaSuccess)
      return nullptr;
    prefer_max_shared(v->fn);
  }
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kShort.fn, kShort.threads,
                                                    kShort.smem(seg_stride(vstride), vstride)) != cudaSuccess)
    return nullptr;
  return (c.nx + kShort.cells - 1) / kShort.cells <= (long)per * sms ? &kShort : &kLong;
}

bool line_shape(Line& L, const kb_config_t& c, const DevState& s) {
  if (s.prec == 0) {
    L.seg = seg64_cells(c.nx, s.sm_count);
    return seg64_prepare();
  }
  L.f32 = line_variant(c, s.g.vstride, s.sm_count);
  if (!L.f32) return false;
  L.seg = L.f32->cells;
  L.smem = L.f32->smem(seg_stride(s.g.vstride), s.g.vstride);
  return true;
}

// the segments' descriptors; ints: nx, ng, nu, nus, vel_off, active, seg_first, nseg, then seg_b and
// seg_i0; longs: cell_off, elem_off; doubles: dx, dt, mu, 1/dx, 1/(2 mu),
// clock[10], respart, FP64 mc64; floats: ul, FP32 mc
static int line_nseg(const kb_config_t& c, int seg) { return (c.nx + seg - 1) / seg; }
static size_t line_doubles(const kb_config_t& c, int seg) { return 18 + 8 * (size_t)line_nseg(c, seg); }
// (8 floats or 4 doubles of Maxwellian coefficients per cell: the same room)
static size_t line_floats(const kb_config_t& c, int ncell) { return (size_t)(c.nu + 3) / 4 * 4 + 8 * (size_t)ncell; }
static size_t line_ints(const kb_config_t& c, int seg) { return 8 + 2 * (size_t)line_nseg(c, seg); }
size_t line_bytes(const kb_config_t& c, int ncell, int seg) {
  return sizeof(SegDesc) * (size_t)line_nseg(c, seg) + 8 * line_doubles(c, seg) + 4 * line_floats(c, ncell) + 4 * line_ints(c, seg);
}

bool line_init(Line& L, const kb_config_t& c, const DevState& s, int ncell, void* mem) {
  const int seg = L.seg;
  const int ns = line_nseg(c, seg);
  SegDesc* G = (SegDesc*)mem;
  double* D = (double*)(G + ns);
  float* F = (float*)(D + line_doubles(c, seg));
  int* I = (int*)(F + line_floats(c, ncell));
  std::vector<double> hd(line_doubles(c, seg), 0.0);
  std::vector<float> hf(line_floats(c, ncell), 0.f);
  std::vector<int> hi(line_ints(c, seg), 0);
  hd[2] = s.g.dx;
  hd[4] = s.g.mu_ref;
  hd[5] = 1.0 / s.g.dx;
  hd[6] = 1.0 / (2.0 * s.g.mu_ref);
  std::vector<double> u(c.nu);
  if (cudaMemcpy(u.data(), s.u, sizeof(double) * c.nu, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
  for (int k = 0; k < c.nu; ++k) hf[k] = float(u[k] - (double)(float)u[k]);
  const int head[8] = {c.nx, c.ngx, c.nu, s.g.vstride, 0, 1, 0, ns};
  for (int k = 0; k < 8; ++k) hi[k] = head[k];
  for (int k = 0; k < ns; ++k) hi[8 + ns + k] = k * seg;  // seg_b stays 0
  std::vector<SegDesc> hg(ns);
  for (int k = 0; k < ns; ++k)
    hg[k] = {0, k * seg, c.nx, c.ngx, c.nu, s.g.vstride, 0, 0, 0, 0, hd[5], float(1.e-7 * s.g.dx), 2.f * float(s.g.mu_ref)};
  if (cudaMemcpy(G, hg.data(), sizeof(SegDesc) * hg.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(D, hd.data(), 8 * hd.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(F, hf.data(), 4 * hf.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(I, hi.data(), 4 * hi.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return false;
  BatchDev& d = L.d;
  d.n = 1;
  d.nx = I;
  d.ng = I + 1;
  d.nu = I + 2;
  d.nus = I + 3;
  d.vel_off = I + 4;
  d.active = I + 5;
  d.seg_first = I + 6;
  d.nseg = I + 7;
  d.seg_b = I + 8;
  d.seg_i0 = I + 8 + ns;
  d.seg_d = G;
  d.cell_off = (const long*)D;
  d.elem_off = (const long*)(D + 1);
  d.dx = D + 2;
  d.dt = D + 3;
  d.mu = D + 4;
  d.rdx = D + 5;
  d.rmu = D + 6;
  d.clock = D + 7;
  d.respart = D + 18;
  d.u = s.u;
  d.wt = s.wt;
  d.uf = s.uf;
  d.wtf = s.wtf;
  d.ul = F;
  d.mc = F + (c.nu + 3) / 4 * 4;
  d.mc64 = (double*)d.mc;
  d.w = s.w;
  d.prim = s.prim;
  d.residual = s.residual;
  d.fw = s.fw;
  d.status = s.status;
  d.nseg_all = ns;
  d.sst_max = seg_stride(s.g.vstride);
  d.nu4_max = s.g.vstride;
  d.K = s.g.K;
  d.gamma = s.g.gamma;
  d.omega = s.g.omega;
  d.Pr = s.g.Pr;
  seg_gas(d);
  d.tol = 0.0;
  d.coll = s.coll;
  L.on = true;
  return true;
}

int line_begin(Line& L, const DevState& s, double dt, cudaStream_t st) {
  if (L.dt != dt) {
    cudaMemcpyAsync((void*)L.d.dt, &dt, sizeof(double), cudaMemcpyHostToDevice, st);
    L.dt = dt;
  }
  if (s.prec == 0) seg64_mcache_launch(L.d, 1, s.ncell, st);
  else seg_mcache_launch(L.d, 1, s.ncell, st);
  return 1;
}

int line_step(Line& L, DevState& s, bool res, int slot, cudaStream_t st, cudaEvent_t mid) {
  const int cur = s.cur;
  cudaError_t e;
  if (s.prec == 0) {
    e = seg64_launch(L.d, L.seg, (const double*)s.h[cur], (const double*)s.b[cur], (double*)s.h[cur ^ 1],
                 (double*)s.b[cur ^ 1], res, slot, st);
  } else {
    const float* hin = (const float*)s.h[cur];
    const float* bin = (const float*)s.b[cur];
    float* hout = (float*)s.h[cur ^ 1];
    float* bout = (float*)s.b[cur ^ 1];
    int want = res;
    void* args[] = {(void*)&L.d, (void*)&hin, (void*)&bin, (void*)&hout, (void*)&bout, (void*)&slot, (void*)&want};
    e = launch_after(L.f32->fn, dim3((unsigned)L.d.nseg_all), dim3((unsigned)L.f32->threads), (size_t)L.smem, st, args);
  }
  if (e != cudaSuccess) return 0;  // the caller's check reports it; the state stays the current one
  s.cur = cur ^ 1;
  if (mid) cudaEventRecord(mid, st);
  if (!res) return 1;
  seg_res_launch(L.d, st);
  return 2;
}

}  // namespace kb
