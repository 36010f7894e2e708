// salsa_chain_taped.cu -- the taped step of the gradient harness.
//
// Bound by the FP64 pipe, mostly in the divisions and roots of the collision kernels and
// their dual-number derivatives; those of salsa_math.cuh are within 0.501 ulp.
// cbrt, exp, log and pow stay CUDA's: with the others the recomputed step moves by some ulps,
// the condensation magnifies them, and the adjoint no longer matches the tangent-linear
// model to 1e-10 (1.6e-10; 3e-13 so).
#define SALSA_MATH_PLAIN_FUNCTIONS
#define SALSA_CHAIN_TAPED
#include "salsa_chain_impl.cuh"

namespace salsa {
const void *chain_taped_entry() { return (const void *)chain_taped_kernel; }
}  // namespace salsa
