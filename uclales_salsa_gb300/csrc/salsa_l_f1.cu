// salsa_l_f1.cu -- instantiation of the step's lane form for KT=float.
#include "salsa_kernel_impl.cuh"

namespace salsa {
cudaError_t launch_lane_f1(const DevParams &P, cudaStream_t st, int grid) {
  return launch_lane_t<float>(P, st, grid);
}
int lane_blocks_per_sm_f1(const DevParams &P) { return lane_blocks_per_sm_t<float>(P); }
}  // namespace salsa
