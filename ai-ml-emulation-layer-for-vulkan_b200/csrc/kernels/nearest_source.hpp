// RESIZE, NEAREST: where an output coordinate comes from (resize.comp:43-134).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mlel {

__host__ __device__ inline int32_t floorDiv(int32_t n, int32_t d) {
    int32_t r = n / d;
    if (r * d > n) {
        --r;
    }
    return r;
}

// Source coordinate along one axis with the shader's 16-bit positions; `pos` is the output coordinate.
__host__ __device__ inline uint32_t nearestSource(uint32_t pos, int32_t n, int32_t d, int32_t offset, uint32_t size) {
    const int32_t y = int32_t(pos * uint32_t(d) + uint32_t(offset));
    const int16_t i = int16_t(floorDiv(y, n));
    const int16_t frac = int16_t(uint32_t(y) - uint32_t(int32_t(i)) * uint32_t(n));
    const int16_t i0 = int16_t(i > 0 ? i : 0);
    const uint32_t next = uint32_t(int32_t(i) + 1);
    const int16_t i1 = int16_t(next < size - 1 ? next : size - 1);
    return uint32_t(int32_t((2 * int32_t(frac) >= n) ? i1 : i0));
}

} // namespace mlel
