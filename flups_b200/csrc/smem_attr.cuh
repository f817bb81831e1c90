// Launch helpers of the line passes: the per-device cache of a kernel's dynamic
// shared-memory attribute, and programmatic launches of chained passes.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace flb {

// cudaFuncSetAttribute(max dynamic shared memory) once per kernel and device:
// the attribute belongs to the device's context, so a process that solves on
// several GPUs sets it on each (one bit per device in `devs`)
template <typename K>
inline cudaError_t smem_attr_once(std::atomic<unsigned long long>& devs, K kernel, size_t smem) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (devs.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) devs.fetch_or(bit, std::memory_order_acq_rel);
    return e;
}

// The passes of one solve follow each other on one stream.  A pass launched
// with chain = 1 is launched when the last block of the pass before it ends,
// instead of after that pass's memory has been flushed and its end reported:
// its blocks set up (addresses, twiddles, Green's values: data no pass writes)
// and wait in pass_begin() until every write of that pass is visible.  2 to 3
// us per gap saved (plain, chained; FP32 free space, HEJ_2, four gaps per solve, and
// the FP64 1500 x 700 plane, two gaps): 64^3 28.7, 20.5 us; 128^3 72.7, 61.5;
// plane 44.4, 39.0; 512^3 3600, 3590, within the scatter of its runs.  Letting
// the next pass start earlier (griddepcontrol.launch_dependents at a pass's
// start) puts its waiting blocks where the last wave has left room and not
// where they would run best: 22.6, 63.5, 46.6 and 3794 us.
__device__ __forceinline__ void pass_begin() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// every kernel launched here calls pass_begin() before it reads or writes what a pass writes
template <typename K, typename A>
inline cudaError_t launch_pass(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t s, const A& args, int chain) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chain ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

}  // namespace flb
