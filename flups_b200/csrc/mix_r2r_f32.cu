// Mixed-radix DCT / DST line passes, f32 (instantiations).
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_r2r_f32(int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    switch (op) {
        case MX_T1: return launch_mix_op<float, MX_T1>(rows, a, ncomp, s);
        case MX_T2: return launch_mix_op<float, MX_T2>(rows, a, ncomp, s);
        case MX_T3: return launch_mix_op<float, MX_T3>(rows, a, ncomp, s);
        default: return launch_mix_op<float, MX_T4>(rows, a, ncomp, s);
    }
}

}  // namespace flb
