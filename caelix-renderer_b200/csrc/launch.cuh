// Launches in a chain: a kernel whose CTAs may start when the last CTA of the kernel before it in the
// stream exits, instead of after that kernel has completed. The kernel calls grid_wait() before it
// touches anything that an earlier command wrote: the wait ends when the kernel before it is complete
// and its writes are visible, and that kernel has waited for the one before it. So the command before a
// chained launch is a kernel of this library that was launched plainly or has waited itself, with nothing
// but event records between the two; after a copy, a memset or a caller's commands the chain starts with
// a plain launch (a caller's kernel may be a dependent one that let its successor start and never waited).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace cx {

__device__ __forceinline__ void grid_wait() { cudaGridDependencySynchronize(); }

// A load of what an earlier kernel of the chain wrote: an ordinary load. The read-only path (__ldg, or a
// const __restrict__ parameter) is for data that no one writes while the kernel exists, and a chained
// kernel exists before the one before it is complete. (Against read-only loads, one B200: the 4,096-leaf build 55
// and 56 us, 2 M grouped leaves 578 and 594.)
template <typename T>
__device__ __forceinline__ T chain_load(const T* p)
{
    return *p;
}

// chained_launch: as above; else a plain launch.
template <typename... Params, typename... Args>
cudaError_t launch_kernel(bool chained_launch, void (*kernel)(Params...), uint32_t grid, uint32_t threads, size_t shared,
                          cudaStream_t stream, Args... args)
{
    cudaLaunchAttribute chained;
    chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chained.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = shared;
    config.stream = stream;
    config.attrs = &chained;
    config.numAttrs = chained_launch ? 1 : 0;
    return cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), uint32_t grid, uint32_t threads, size_t shared, cudaStream_t stream,
                           Args... args)
{
    return launch_kernel(true, kernel, grid, threads, shared, stream, args...);
}

}  // namespace cx
