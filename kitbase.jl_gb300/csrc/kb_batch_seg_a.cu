// Instantiations of the fused FP32 batch segment kernel (kb_batch.cuh), split
// across translation units so that they compile in parallel.
#include "kb_batch.cuh"

namespace kb {

void seg_variants_a(std::vector<SegVariant>& out) {
  out.push_back({8, 64, 7, (const void*)k_batch_seg<7, 64>, seg_smem<7, 64>, seg_smem_max<7, 64>()});
  out.push_back({16, 64, 15, (const void*)k_batch_seg<15, 64>, seg_smem<15, 64>, seg_smem_max<15, 64>()});
  out.push_back({16, 128, 15, (const void*)k_batch_seg<15, 128>, seg_smem<15, 128>, seg_smem_max<15, 128>()});
  out.push_back({16, 256, 15, (const void*)k_batch_seg<15, 256>, seg_smem<15, 256>, seg_smem_max<15, 256>()});
}

}  // namespace kb
