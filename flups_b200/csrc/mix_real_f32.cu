// Mixed-radix real-to-complex and complex-to-real line passes, f32 (instantiations).
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_real_f32(int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    if (op == MX_R2C) return launch_mix_op<float, MX_R2C>(rows, a, ncomp, s);
    return launch_mix_op<float, MX_C2R>(rows, a, ncomp, s);
}

}  // namespace flb
