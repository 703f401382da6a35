// launch.cuh -- launches that overlap the end of the kernel before them.
//
// A call is a chain of short kernels on one stream.  A kernel launched by
// launch_after starts as soon as every block of the kernel before it has
// started and passed after_previous (programmatic dependent launch): its launch
// and its prologue overlap that kernel, and after_previous holds it until that
// kernel has finished and its writes can be read.  Kernels that such a launch
// follows, and those launched so, call after_previous before they read or write
// global memory; launched the usual way, or behind anything but a kernel, the
// call returns at once.
#pragma once

#include <cuda_runtime.h>

namespace gsc {

__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

// after_previous in two steps, for a kernel of few blocks before one that fills
// the GPU: wait_previous, then next_may_start at the end.  Blocks of the next
// kernel that came earlier would find SMs partly taken, and run as a wave of
// their own.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace gsc
