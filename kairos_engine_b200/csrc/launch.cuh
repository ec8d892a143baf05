/* launch.cuh — kernel launches with programmatic dependent launch: the next kernel of the stream may be made resident, and
 * run up to its sp_pdl_wait(), while this one drains. A kernel launched with sp_launch calls sp_pdl_wait() in every thread
 * before it touches anything an earlier kernel wrote or still reads. */
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void sp_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void sp_pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t sp_launch(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, int *nl, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    (*nl)++;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
