// Launches with programmatic stream serialization: a kernel's CTAs take their places while the one before it on the stream drains.
// Every kernel launched so waits (`wait_for_previous`) before it reads or writes anything that others may have written or
// may still read; its own successor is let in from `let_next_in` on, and waits in turn until this kernel is complete.  A kernel without
// `let_next_in` has it in as its CTAs leave.
//
// Two kernels read before they wait: the products of the channel mixer request tiles of the weights, the chunk gradients of the training step
// tiles of the sequence and the output's gradient.  That is sound only behind a kernel of the same call that writes none of it and itself
// calls `wait_for_previous` before `let_next_in`: whatever wrote those tensors is complete when such a kernel lets its successor in.  A
// kernel that lets its successor in before it has waited must not be put in front of them.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace rwkv7 {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// (a kernel of clusters has their size in its declaration)
template <typename... Params, typename... Args>
cudaError_t launch_serialized(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e == cudaSuccess) count_launch();
    return e;
}

}  // namespace rwkv7
