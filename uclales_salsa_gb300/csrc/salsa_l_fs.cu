// salsa_l_fs.cu -- instantiation of the step's lane form for KT=float, with secondary ice.
#include "salsa_kernel_impl.cuh"

namespace salsa {
cudaError_t launch_lane_fs(const DevParams &P, cudaStream_t st, int grid) {
  return launch_lane_t<float, true>(P, st, grid);
}
int lane_blocks_per_sm_fs(const DevParams &P) { return lane_blocks_per_sm_t<float, true>(P); }
}  // namespace salsa
