#pragma once

#include <cuda_runtime.h>

namespace fwi {

// FP32 to FP64 by integer operations, exact for every value (denormals by way of 2^64 times them): the
// conversion instruction runs on the FP64 pipe, 64 cycles a warp on an SM quarter.
__device__ __forceinline__ double widen(float v)
{
    unsigned u = __float_as_uint(v), a = u & 0x7fffffffu;
    unsigned bias = a >= 0x7f800000u ? 0x70000000u : 0x38000000u;  // added to the shifted exponent: inf and NaN keep all ones
    if (a < 0x00800000u) {
        u = __float_as_uint(v * 0x1p64f);
        a = u & 0x7fffffffu;
        bias = 0x38000000u - (64u << 20);
    }
    return __hiloint2double((int)((u & 0x80000000u) | (a ? (a >> 3) + bias : 0u)), (int)(u << 29));
}
__device__ __forceinline__ double widen(double v) { return v; }

}  // namespace fwi
