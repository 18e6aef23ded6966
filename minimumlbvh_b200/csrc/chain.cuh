// Kernels launched as a chain: each may start while the one before it drains
// (programmatic dependent launch), which hides its launch latency. Every
// kernel of a chain calls chain_begin() in all threads before it touches
// memory: it lets the next kernel start and waits until the one before is
// complete and its writes are visible. A kernel only completes after its own
// wait, so completion is transitive along the chain.
#pragma once

#include <cuda_runtime.h>

namespace mlbvh {

__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches a kernel that follows another kernel of its chain on the stream.
// The first kernel of a chain is launched as any other.
template <class... Params, class... Args>
inline void launch_chained(void (*kernel)(Params...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t stream,
                           Args... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);  // errors: MLBVH_CHECK_LAUNCH
}

}  // namespace mlbvh
