// salsa_l_ds.cu -- instantiation of the step's lane form for KT=double, with secondary ice.
#include "salsa_kernel_impl.cuh"

namespace salsa {
cudaError_t launch_lane_ds(const DevParams &P, cudaStream_t st, int grid) {
  return launch_lane_t<double, true>(P, st, grid);
}
int lane_blocks_per_sm_ds(const DevParams &P) { return lane_blocks_per_sm_t<double, true>(P); }
}  // namespace salsa
