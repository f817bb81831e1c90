// Mixed-radix fused ROT line passes (instantiations).  One launch per field: the
// three components of a line position are the CTA's.
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_rot(int f64, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    if (ncomp != 3) return cudaErrorInvalidValue;
    return f64 ? launch_mix_op<double, MX_ROT>(rows, a, 1, s) : launch_mix_op<float, MX_ROT>(rows, a, 1, s);
}

}  // namespace flb
