// salsa_l_d1.cu -- instantiation of the step's lane form for KT=double.
#include "salsa_kernel_impl.cuh"

namespace salsa {
cudaError_t launch_lane_d1(const DevParams &P, cudaStream_t st, int grid) {
  return launch_lane_t<double>(P, st, grid);
}
int lane_blocks_per_sm_d1(const DevParams &P) { return lane_blocks_per_sm_t<double>(P); }
}  // namespace salsa
