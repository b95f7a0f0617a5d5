// pdl.cuh -- launches that overlap their start with the end of the kernel
// before them on the stream (programmatic dependent launch).  For sequences of
// short kernels: the next grid is set up while the last one drains, and each
// kernel waits (pdl_wait) for the one before it to complete, with its writes
// visible, before it touches memory.
//
// A grid of the sequence can be resident while the grid two before it still
// runs, so what the others write changes during its own lifetime.  Such a
// kernel takes no const __restrict__ pointers: the compiler may read those
// through the non-coherent path, which is defined only for memory that nobody
// writes while the kernel runs.  Plain loads behind pdl_wait see the writes.
// (Reading through the L2 only, by __ldcg, costs the greedy steps 9 % and the
// rounds of 2^24 entries 1-2 %.)
#pragma once
#include <cuda_runtime.h>

// First statements of a kernel launched with launch_pdl.
__device__ __forceinline__ void pdl_wait() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t stream, A... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
