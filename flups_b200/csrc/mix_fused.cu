// Mixed-radix fused line passes: forward DFT, Green's multiply, inverse DFT (instantiations).
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_fused(int f64, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    return f64 ? launch_mix_op<double, MX_FUSED>(rows, a, ncomp, s) : launch_mix_op<float, MX_FUSED>(rows, a, ncomp, s);
}

}  // namespace flb
