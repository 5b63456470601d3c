// split_launch.cuh -- launches of split_kernel.
#pragma once
#include <algorithm>

#include "split_kernel.cuh"

namespace tis {

inline void split_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int nlane, int nsplit, int nt, size_t smem,
                         cudaStream_t st) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(nsplit * nlane, 1, 1);
  cfg.blockDim = dim3(nt, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = nsplit; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
}

template <typename Real, int NT, bool PER>
cudaError_t split_run(int nlane, size_t smem, cudaStream_t st, const KArgs &a) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  split_config(cfg, at, nlane, a.nsplit, NT, smem, st);
  if (a.ew_nwork) {   // lanes and workers wait for one another: all resident, or an error
    cfg.gridDim.x += a.ew_nwork;
    cfg.dynamicSmemBytes = std::max<size_t>(smem, ew_smem(a.nlane, a.ew_nqmax, a.ew_ncol).total);
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, split_kernel<Real, NT, PER>, a);
}

// allows the kernel all the shared memory a CTA may have (contexts of
// different sizes share it) and clusters beyond the portable 8; gives how
// many clusters of nsplit CTAs with smem bytes each the GPU holds at once
template <typename Real, int NT, bool PER>
cudaError_t split_prepare(int nsplit, size_t smem, int *clusters) {
  auto k = split_kernel<Real, NT, PER>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e == cudaSuccess && nsplit > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[1];
  split_config(cfg, at, 1, nsplit, NT, smem, nullptr);
  return cudaOccupancyMaxActiveClusters(clusters, k, &cfg);
}

} // namespace tis
