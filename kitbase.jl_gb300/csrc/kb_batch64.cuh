// kb_batch64.cuh -- launch interface of the FP64 segment kernel
// (kb_batch64.cu) of the batched and single 1D2F1V solves.
#pragma once

#include "kb_batch.cuh"

namespace kb {

constexpr int SEG64_MAX = 8;  // most cells per segment

// Cells per segment for `cells` cells in all on a GPU of `sms` multiprocessors.
int seg64_cells(long cells, int sms);
// Dynamic shared memory of a CTA of segments of `seg` cells, rows of at most
// `ns` values.
int seg64_smem(int seg, int ns);
// Raise the kernel's shared-memory limit on the current device (outside any
// stream capture).  False when the device refuses.
bool seg64_prepare();
// One step of every segment (B.nseg_all CTAs).  want_res: leave the segments'
// residual sums in B.respart, and their face moments where B.fw is given.  slot:
// see BatchDev::clock (-1: dt from B.dt).
cudaError_t seg64_launch(const BatchDev& B, int seg, const double* hin, const double* bin, double* hout,
                         double* bout, bool want_res, int slot, cudaStream_t st);
// Per-instance residual of the last step that left its sums (k_batch_seg_res).
void seg_res_launch(const BatchDev& B, cudaStream_t st);
// Maxwellian coefficients of every cell from its prim (BatchDev::mc64, mc).
void seg64_mcache_launch(const BatchDev& B, int n, int max_cells, cudaStream_t st);
void seg_mcache_launch(const BatchDev& B, int n, int max_cells, cudaStream_t st, int b0 = 0);

}  // namespace kb
