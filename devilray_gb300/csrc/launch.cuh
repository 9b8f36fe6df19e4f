// launch.cuh -- programmatic dependent launch of kernels that follow one another
// in a stream.
//
// A kernel launched with launch_after() may start once every block of the kernel
// before it in the stream has called allow_next() (or ended); it must call
// wait_previous() before it touches memory that any earlier kernel of the stream
// reads or writes. wait_previous() returns when the kernel before it is complete
// and its stores are visible; as every kernel of a chain waits, all earlier ones
// are complete too. What overlaps is the launch itself and the part of a kernel
// before the wait (about 2 us per launch). In a kernel launched the ordinary way
// both calls do nothing.
#pragma once

#include <cuda_runtime.h>

namespace dr {

__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `early` = false: the ordinary launch, for callers that choose by their stream.
template <typename... P, typename... A>
cudaError_t launch_next(bool early, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args)
{
    return launch_next(true, kernel, grid, block, smem, st, args...);
}

}  // namespace dr
