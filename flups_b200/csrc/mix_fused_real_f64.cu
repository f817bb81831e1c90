// Mixed-radix fused passes of a real last direction, f64 (instantiations).
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_fused_real_f64(int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    switch (op) {
        case MX_FUSED_R: return launch_mix_op<double, MX_FUSED_R>(rows, a, ncomp, s);
        case MX_FUSED_23: return launch_mix_op<double, MX_FUSED_23>(rows, a, ncomp, s);
        case MX_FUSED_32: return launch_mix_op<double, MX_FUSED_32>(rows, a, ncomp, s);
        case MX_FUSED_11: return launch_mix_op<double, MX_FUSED_11>(rows, a, ncomp, s);
        default: return launch_mix_op<double, MX_FUSED_44>(rows, a, ncomp, s);
    }
}

}  // namespace flb
