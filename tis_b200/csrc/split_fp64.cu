// split_fp64.cu -- split_kernel for FP64 lanes (one unit
// per variant: they compile side by side).
#include "split_launch.cuh"

namespace tis {

cudaError_t split_launch_fp64(int nlane, int nt, size_t smem, cudaStream_t st, const KArgs &a) {
  return nt == 256 ? split_run<double, 256, false>(nlane, smem, st, a) : split_run<double, 512, false>(nlane, smem, st, a);
}

cudaError_t split_setup_fp64(int nsplit, int nt, size_t smem, int *clusters) {
  return nt == 256 ? split_prepare<double, 256, false>(nsplit, smem, clusters) : split_prepare<double, 512, false>(nsplit, smem, clusters);
}

} // namespace tis
