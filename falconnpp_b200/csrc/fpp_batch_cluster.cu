// fpp_batch_cluster.cu — instances of the one-query-per-cluster kernel for
// small batches (k_cluster_query): BF16, FP8 and the int8-screened FP32 form.
#include "fpp_batch_kernel.cuh"

namespace fpp {

template <int MODE, int VI32>
static KernelSel cluster_ptr() {
  const void* fn = reinterpret_cast<const void*>(&k_cluster_query<MODE, VI32>);
  const size_t smem = BatchSmem<kBThreads / 8>::kBytes;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return KernelSel{fn, smem};
}

template <int MODE>
static KernelSel cluster_mode(int v32) {
  if (v32 == 1) return cluster_ptr<MODE, 1>();
  if (v32 == 2) return cluster_ptr<MODE, 2>();
  return cluster_ptr<MODE, 4>();
}

KernelSel pick_kernel_cluster(int mode, int d) {
  const int v32 = vi_of(d, 4);
  if (mode == kRowsI8) return cluster_mode<kRowsI8>(v32);
  if (mode == kRowsBF16) return cluster_mode<kRowsBF16>(v32);
  if (mode == kRowsFP8) return cluster_mode<kRowsFP8>(v32);
  return KernelSel{nullptr, 0};
}

}  // namespace fpp
