// Launches with programmatic stream serialization: a kernel's CTAs take their places while the one before it on the stream drains.
// Every kernel launched so waits (`wait_for_previous`) before it reads or writes anything that others may have written or
// may still read; its own successor is let in from `let_next_in` on, and waits in turn until this kernel is complete.
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace rwkv7 {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

template <typename... Params, typename... Args>
cudaError_t launch_serialized_cluster(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem, unsigned cluster, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e == cudaSuccess) count_launch();
    return e;
}
// (a kernel with its cluster size in its declaration, or none)
template <typename... Params, typename... Args>
cudaError_t launch_serialized(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, Args... args) {
    return launch_serialized_cluster(kernel, grid, threads, smem, 1u, stream, args...);
}

}  // namespace rwkv7
