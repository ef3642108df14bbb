// Launches that overlap their start with the end of the kernel before them on
// the stream (programmatic dependent launch): the next kernel's blocks are put
// on the chip while the last ones of this kernel run, and wait there.
#pragma once

#include <cuda_runtime.h>

namespace bj {

// First statement of a kernel launched with launch_after, for every thread:
// returns when the kernels before this one are complete and their writes
// visible, and lets the kernel after this one be put on the chip once all
// blocks of this one are there. (Launched the usual way it does nothing.)
__device__ __forceinline__ void begin_after_previous() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

// The launch's status: a refused launch is reported here and nowhere else.
template <typename... P, typename... A>
[[nodiscard]] cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute overlap{};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &overlap;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

} // namespace bj
