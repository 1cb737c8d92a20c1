// kb_line.cuh -- single 1D2F1V solves stepped by the fused segment kernels of
// the batch (kb_line.cu).
#pragma once

#include "../../include/kitgpu.h"
#include "kb_batch64.cuh"

namespace kb {

// Device tables that present one handle's solve to the segment kernels as a
// batch of one, and the chosen segment kernel.
struct Line {
  bool on = false;
  BatchDev d;
  int seg = 0;                 // cells per segment
  const SegVariant* f32 = nullptr;  // FP32 kernel
  int smem = 0;
  double dt = 0.0;             // time step held by d.dt
};

// The solves the segment kernels cover: 1D2F1V, KFVS, fixed ends, van Leer,
// at most 256 velocities.
bool line_covers(const kb_config_t& c);
// Choose the segment kernel and its cells per segment (L.seg, L.f32, L.smem);
// outside any capture.
bool line_shape(Line& L, const kb_config_t& c, const DevState& s);
// Bytes of one allocation for the tables of nx cells (ncell incl. ghosts)
size_t line_bytes(const kb_config_t& c, int ncell, int seg);
// Fill `mem` (line_bytes) and L for the solve in s, after line_shape; u: the
// host's velocities.
bool line_init(Line& L, const kb_config_t& c, const DevState& s, const double* u, int ncell, void* mem);
// Before steps with time step dt (outside any capture): the step in device
// memory and the Maxwellian coefficients of the current prim.  Returns the
// number of launches.
int line_begin(Line& L, const DevState& s, double dt, cudaStream_t st);
// One step (advances s.cur); res: with its residual.  slot: BatchDev::clock.
// mid: recorded between the step's kernel and the residual's.
int line_step(Line& L, DevState& s, bool res, int slot, cudaStream_t st, cudaEvent_t mid = nullptr);

}  // namespace kb
