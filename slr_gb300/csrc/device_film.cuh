// From a colour value of the film to its byte (sRGB gamma, spectrum_base.cpp:16-21).
#pragma once
#include <cstdint>

namespace slrgpu {

__device__ __forceinline__ float srgbGamma(float v) {
    if ((double)v <= 0.0031308) return (float)__dmul_rn(12.92, (double)v);
    return (float)__dsub_rn(__dmul_rn(1.055, pow((double)v, 1.0 / 2.4)), 0.055);
}

// min(255, 256 x gamma(v)) as an integer.  The gamma's power is taken in single
// precision first: powf is within 4 units in the last place (CUDA's stated
// bound) and its exponent within half a unit, so 256 x gamma is off by less
// than 2e-4; only a value within 1e-3 of an integer, where that could matter,
// takes the double-precision power, whose result decides every such byte.
// (FP64 is a 64th of this chip's FP32 rate: three double powers per pixel took
// 1.4 ms of a 1920 x 1080 film's 2.9 ms.)
__device__ __forceinline__ uint8_t srgbByte(float v) {
    if ((double)v > 0.0031308) {
        const float x = 256.0f * (1.055f * powf(v, (float)(1.0 / 2.4)) - 0.055f);
        if (fabsf(x - rintf(x)) >= 1e-3f) return (uint8_t)min(255u, (uint32_t)x);
    }
    return (uint8_t)min(255u, (uint32_t)__fmul_rn(256.0f, srgbGamma(v)));
}

}  // namespace slrgpu
