// split_mixed.cu -- split_kernel for mixed-precision lanes (one unit
// per variant: they compile side by side).
#include "split_launch.cuh"

namespace tis {

cudaError_t split_launch_mixed(int nlane, int nt, size_t smem, cudaStream_t st, const KArgs &a) {
  return nt == 256 ? split_run<float, 256, false>(nlane, smem, st, a) : split_run<float, 512, false>(nlane, smem, st, a);
}

cudaError_t split_setup_mixed(int nsplit, int nt, size_t smem, int *clusters) {
  return nt == 256 ? split_prepare<float, 256, false>(nsplit, smem, clusters) : split_prepare<float, 512, false>(nsplit, smem, clusters);
}

} // namespace tis
