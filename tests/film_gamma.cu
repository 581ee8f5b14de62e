/* Every float of [lo, hi] through the film's byte function and through the
 * double-precision gamma alone: how many bytes differ, and how many would if the
 * single-precision power decided all of them. */
#include "../slr_gb300/csrc/device_film.cuh"

using namespace slrgpu;

__global__ void kCompare(uint32_t lo, uint32_t hi, unsigned long long* counts) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long u = lo + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; u <= hi; u += step) {
        const float v = __uint_as_float((uint32_t)u);
        const uint8_t want = (uint8_t)min(255u, (uint32_t)__fmul_rn(256.0f, srgbGamma(v)));
        if (srgbByte(v) != want) atomicAdd(counts, 1ull);
        const float x = 256.0f * (1.055f * powf(v, (float)(1.0 / 2.4)) - 0.055f);
        if ((double)v > 0.0031308 && (uint8_t)min(255u, (uint32_t)x) != want) atomicAdd(counts + 1, 1ull);
    }
}

extern "C" int film_gamma_compare(uint32_t lo, uint32_t hi, unsigned long long counts[2]) {
    unsigned long long* dev = nullptr;
    cudaError_t e = cudaMalloc(&dev, 2 * sizeof(*dev));
    if (e == cudaSuccess) e = cudaMemset(dev, 0, 2 * sizeof(*dev));
    if (e == cudaSuccess) {
        kCompare<<<1216, 256>>>(lo, hi, dev);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(counts, dev, 2 * sizeof(*dev), cudaMemcpyDeviceToHost);
    cudaFree(dev);
    return (int)e;
}
