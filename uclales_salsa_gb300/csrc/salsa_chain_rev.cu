// salsa_chain_rev.cu -- the reverse step of the gradient harness.
//
// Bound by the FP64 pipe.  It is linear in the adjoint and recomputes only local partial
// derivatives of the taped states, so it takes all of salsa_math.cuh.  Forward and adjoint of
// 8,192 cells x 8 steps: 88.0 ms with plain operations throughout, 84.6 with these in the
// reverse step, 78.8 with the divisions and roots of the taped step too.
#define SALSA_CHAIN_REVERSE
#include "salsa_chain_impl.cuh"

namespace salsa {
const void *chain_rev_entry() { return (const void *)chain_rev_kernel; }
}  // namespace salsa
