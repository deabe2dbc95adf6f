// ens_kernel.cuh -- the persistent ensemble kernel (persistent.cuh) and its
// launch entry points, included by one translation unit per precision: the
// kernel inlines every pass body of every grid size it supports.
#pragma once
#define DNSB_PERSISTENT_KERNELS
#include "persistent.cuh"

namespace dnsb {

template <class R>
cudaError_t p_prepare(size_t smem, int *blocks_per_sm) {
  cudaError_t e = cudaFuncSetAttribute(k_ens_step<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_ens_step<R>, PBS, smem);
}

// one cooperative launch (all blocks co-resident, or the launch fails)
template <class R>
cudaError_t p_launch(int grid, size_t smem, cudaStream_t st, const PPlan<R> *plan, PSync *sy,
                     unsigned long long wait_ns) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(PBS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_ens_step<R>, plan, sy, wait_ns);
}

}  // namespace dnsb
