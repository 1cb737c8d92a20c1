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

// One allocation: the tables that kb_create uploads in one copy (the FP32 kernel's
// descriptors, head, ul, ints), then the residual's sums and the Maxwellian
// coefficients.
struct LineHead {
  long cell_off, elem_off;
  double dx, dt, rdx, rmu, clock[10];
};
static_assert(sizeof(LineHead) % 16 == 0, "what follows is read by 16 bytes");
struct LinePlan {
  int ns;  // segments
  size_t head, ul, ints, copy, respart, mc, total;  // byte offsets; copy: bytes uploaded
  LinePlan(const kb_config_t& c, int ncell, int seg) {
    const auto up = [](size_t x) { return (x + 15) / 16 * 16; };
    ns = (c.nx + seg - 1) / seg;
    head = c.precision == KB_PREC_FP64 ? 0 : sizeof(SegDesc) * (size_t)ns;
    ul = head + sizeof(LineHead);
    ints = up(ul + 4 * (size_t)c.nu);
    copy = ints + 4 * (8 + (c.precision == KB_PREC_FP64 ? 2 * (size_t)ns : 0));  // nx, ng, nu, nus, vel_off, active,
    respart = up(copy);                                                          // seg_first, nseg; FP64: seg_b, seg_i0
    mc = respart + 64 * (size_t)ns;
    total = mc + 32 * (size_t)ncell;  // 8 floats or 4 doubles of coefficients per cell
  }
};
size_t line_bytes(const kb_config_t& c, int ncell, int seg) { return LinePlan(c, ncell, seg).total; }

bool line_init(Line& L, const kb_config_t& c, const DevState& s, const double* u, int ncell, void* mem) {
  const LinePlan P(c, ncell, L.seg);
  const int ns = P.ns, seg = L.seg;
  std::vector<char> host(P.copy, 0);
  LineHead& H = *(LineHead*)(host.data() + P.head);
  H.dx = s.g.dx;
  H.rdx = 1.0 / s.g.dx;
  H.rmu = 1.0 / (2.0 * s.g.mu_ref);
  float* hf = (float*)(host.data() + P.ul);
  for (int k = 0; k < c.nu; ++k) hf[k] = float(u[k] - (double)(float)u[k]);
  int* hi = (int*)(host.data() + P.ints);
  const int head[8] = {c.nx, c.ngx, c.nu, s.g.vstride, 0, 1, 0, ns};
  for (int k = 0; k < 8; ++k) hi[k] = head[k];
  if (s.prec == 0) {
    for (int k = 0; k < ns; ++k) hi[8 + ns + k] = k * seg;  // seg_b stays 0
  } else {
    SegDesc* G = (SegDesc*)host.data();
    for (int k = 0; k < ns; ++k)
      G[k] = {0, k * seg, c.nx, c.ngx, c.nu, s.g.vstride, 0, 0, 0, 0, H.rdx, float(1.e-7 * s.g.dx), 2.f * float(s.g.mu_ref)};
  }
  char* M = (char*)mem;
  if (cudaMemcpy(M, host.data(), P.copy, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(M + P.respart, 0, 64 * (size_t)ns) != cudaSuccess)
    return false;
  const LineHead* D = (const LineHead*)(M + P.head);
  int* I = (int*)(M + P.ints);
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
  d.seg_d = (const SegDesc*)M;
  d.cell_off = &D->cell_off;
  d.elem_off = &D->elem_off;
  d.dx = &D->dx;
  d.dt = &D->dt;
  d.rdx = &D->rdx;
  d.rmu = &D->rmu;
  d.clock = (double*)D->clock;
  d.respart = (double*)(M + P.respart);
  d.u = s.u;
  d.wt = s.wt;
  d.uf = s.uf;
  d.wtf = s.wtf;
  d.ul = (const float*)(M + P.ul);
  d.mc = (float*)(M + P.mc);
  d.mc64 = (double*)(M + P.mc);
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
