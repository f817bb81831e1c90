// One operation of the mixed-radix passes in one precision and line direction:
// FLB_MIX_OP (MixOp), FLB_MIX_T (float, double) and FLB_MIX_ROWS (true, false)
// come from the build, which compiles this file once for each of them.  A
// module is loaded whole when its first kernel runs, and the line tables are
// most of it: with the eight FP64 DCT / DST kernels in one module that took 10
// ms.  First solve of a process, ten modules -> sixty: 250 x 150 x 180 box
// (FP64) 30 -> 4.5 ms, 145 x 121 x 101 node grid (FP32) 11.6 -> 6.1, 200^3
// (FP64) 9.4 -> 4.3, 1500 x 700 plane 7.3 -> 3.0.
#include "mix_dft_impl.cuh"

#if !defined(FLB_MIX_OP) || !defined(FLB_MIX_T) || !defined(FLB_MIX_ROWS)
#error "mix_unit.cu is compiled once per operation, precision and direction (flups_b200/build.py)"
#endif

namespace flb {

template cudaError_t launch_mix_op<FLB_MIX_T, FLB_MIX_OP, FLB_MIX_ROWS>(const MixArgs& a, int ncomp, cudaStream_t s);

}  // namespace flb
