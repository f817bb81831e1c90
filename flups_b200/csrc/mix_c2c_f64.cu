// Mixed-radix complex line passes, f64 (instantiations).
#include "mix_dft_impl.cuh"

namespace flb {

cudaError_t launch_mix_c2c_f64(int op, bool rows, const MixArgs& a, int ncomp, cudaStream_t s) {
    if (op == MX_C2C_F) return launch_mix_op<double, MX_C2C_F>(rows, a, ncomp, s);
    return launch_mix_op<double, MX_C2C_I>(rows, a, ncomp, s);
}

}  // namespace flb
