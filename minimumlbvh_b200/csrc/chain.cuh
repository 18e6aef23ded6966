// Kernels launched as a chain: each may start while the one before it drains
// (programmatic dependent launch), which hides its launch latency. Every
// kernel of a chain calls chain_begin() in all threads before it touches
// memory: it lets the next kernel start and waits until the one before is
// complete and its writes are visible. A kernel only completes after its own
// wait, so completion is transitive along the chain.
//
// What an earlier kernel of the chain wrote is read with chain_load. The
// read-only path (__ldg, or a `const T* __restrict__` parameter, whose loads
// the compiler may send there) is for data that nothing writes while the kernel
// is resident, which here begins before its predecessors end: it is kept for
// the chain's inputs, the triangles and the mesh offsets.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mlbvh {

__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// An ordinary load: chain_begin's wait makes what earlier kernels wrote visible
// to it, and its memory clobber keeps the compiler from moving it up. Whole
// builds of 1,000 / 213,000 / 4M triangles: 20.9 / 80.6 / 517 us; loads pinned
// to the L2 by volatile assembly 24.6 / 87.4 / 528, the read-only path 22.5 /
// 84.9 / 529.
template <class T>
__device__ __forceinline__ T chain_load(const T* p)
{
    return *p;
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
