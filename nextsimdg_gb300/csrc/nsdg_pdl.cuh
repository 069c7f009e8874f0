// nsdg_pdl.cuh — the order between a sub-cycle's launches.
//
// Stress and node kernels alternate, each launched as a programmatic dependent
// of the one before: its blocks start when every block of that kernel has
// passed its own wait (waitForPrevious lets the next launch go right there),
// so they load the step's constants, and what the kernel before that one wrote,
// while it still runs.  A kernel may therefore read before its wait only what
// the launch directly before it does not write, and write nothing.
//
// Update of 100 iterations, the next launch at the wait against at the end: mixed
// mEVP 64 x 64 0.44 against 0.48 ms, 256 x 256 0.83 against 0.90, BBM 64 x 64 0.72
// against 0.79, 192 x 192 1.18 against 1.42.  The FP64 kernels are bound by the
// SM's FP64 unit: blocks that start while others run land unevenly, and with two
// to four blocks per SM that costs more than it gives (mEVP 96 x 96
// quadrilaterals 1.41 against 1.27, BBM 96 x 96 4.3 against 2.9), so they let the
// next launch go early only where releaseEarly64 says so, the BBM ones never.
//
//   before the wait: arrays that the sub-cycle changes are read from L2
//     (their writer had finished when the launch before passed its wait; a line
//     of an L1 may be older);
//   after it: as ordinary global loads (not through the read-only path, which
//     takes memory that does not change while a kernel lives).
//
// A launch that follows another one of the same kernel (nsdg_kernel_time_kernel)
// has no such order: it is an ordinary one (programmatic = false).
#pragma once

#include <cuda_runtime.h>

namespace nsdg {
namespace {

template <typename... KArgs, typename... Args>
cudaError_t launchAfter(bool programmatic, cudaStream_t s, void (*kernel)(KArgs...), size_t blocks, int threads,
    size_t shared, Args... args)
{
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__device__ __forceinline__ void waitForPrevious(bool release = true)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (release)
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename T> __device__ __forceinline__ T beforeWait(const T* p) { return __ldcg(p); }
__device__ __forceinline__ float afterWait(const float* p)
{
    float x;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ double afterWait(const double* p)
{
    double x;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(p));
    return x;
}

} // namespace
} // namespace nsdg
