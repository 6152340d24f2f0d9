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

// FP64 to FP32, rounded to nearest even as the conversion does, by integer operations where the result is
// zero or a normal number; the rest converts (out of line: as a branch the compiler would run it for
// every value).
static __device__ __noinline__ float narrow_any(double v) { return (float)v; }
template <typename T> __device__ __forceinline__ T narrow(double v);
template <> __device__ __forceinline__ double narrow<double>(double v) { return v; }
template <> __device__ __forceinline__ float narrow<float>(double v)
{
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v), m = hi & 0x7fffffffu;
    const unsigned b = (m - 0x38000000u) << 3 | lo >> 29, rest = lo & 0x1fffffffu;  // 23 bits kept, 29 dropped
    const unsigned r = b + (rest + (b & 1u) > 0x10000000u ? 1u : 0u);               // (a carry moves into the exponent)
    if (m - 0x38100000u < 0x47f00000u - 0x38100000u) return __uint_as_float((hi & 0x80000000u) | r);
    return (m | lo) == 0u ? __uint_as_float(hi) : narrow_any(v);
}

}  // namespace fwi
