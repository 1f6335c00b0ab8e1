// Launches whose start overlaps the end of the kernel in front of them in the stream (programmatic dependent launch).
//
// A kernel of a small problem runs for 3 to 10 us, and between two such kernels in a stream the device idles for a
// microsecond or more: the second launch is only set up once the first kernel has ended.  With this attribute its
// blocks are set up, and run up to grid_dependency_wait, as soon as all blocks of the first kernel have left.
// Every kernel launched this way waits before it touches global memory, so the order of memory accesses in the
// stream is as before.  (The kernels do not ask for the next one earlier than that: blocks that wait beside those of
// the kernel in front of them take their places unevenly, 2558 x 626 SpMM with N = 24 11.3 -> 18.4 us, masked SDDMM
// 8192 x 8192, inner dimension 64 91 -> 112 us.)
#pragma once
#include <cuda_runtime.h>

namespace dlspm {

// Work of the kernels in front in the stream is complete and visible from here on.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The next launch in the stream may be set up from here on (by default: from the end of the block on).
__device__ __forceinline__ void grid_dependency_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches `kernel` (which begins with grid_dependency_wait); errors are left for cudaGetLastError.
template <typename... Params, typename... Args>
inline void launch_overlapped(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t shared, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace dlspm
