// bits.cuh -- bit scans for device and host code.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace dr {

__host__ __device__ __forceinline__ int lowest_bit(uint32_t m)
{
#if defined(__CUDA_ARCH__)
    return __ffs(m) - 1;
#else
    return __builtin_ctz(m);
#endif
}

__host__ __device__ __forceinline__ int popcount(uint32_t m)
{
#if defined(__CUDA_ARCH__)
    return __popc(m);
#else
    return __builtin_popcount(m);
#endif
}

}  // namespace dr
