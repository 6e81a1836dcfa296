// Programmatic dependent launch for chains of short kernels: a kernel launched
// with launch_next may be set up and its CTAs placed while the kernel before it
// in the stream still runs; pdl_begin, its first statement, lets the kernel
// after it do the same and then waits until everything before has finished and
// its writes are visible.  Kernels of a few microseconds otherwise spend as
// long between each other as in each other.  Such a kernel reads through plain
// pointers (no __restrict__, no __ldg): a load from memory that the compiler
// takes for constant could move above the wait.
#pragma once
#include <cuda_runtime.h>

namespace rfx {

__device__ __forceinline__ void pdl_begin() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

template <typename... Params, typename... Args>
cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace rfx
