// The split of a ray query's rays over the blocks of its kernel, and a warp's
// step through the rays of its block.  Plain arithmetic, for the kernel and for
// the host test that walks it.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SLRGPU_HD __host__ __device__ __forceinline__
#else
#define SLRGPU_HD inline
#endif

namespace slrgpu {

// Block `block` of `blocks` takes the `count` rays from `first` on.
struct RayBlock {
    uint32_t first, count;
};
SLRGPU_HD uint64_t raysPerBlock(uint32_t n, uint32_t blocks) { return ((uint64_t)n + blocks - 1) / blocks; }
SLRGPU_HD RayBlock rayBlock(uint32_t n, uint32_t blocks, uint32_t block) {
    const uint64_t chunk = raysPerBlock(n, blocks), first = chunk * block;
    if (first >= n) return RayBlock{n, 0};
    return RayBlock{(uint32_t)first, (uint32_t)(n - first < chunk ? n - first : chunk)};
}

// The block's cursor counts the rays its warps have asked for, from 0: each asks
// at most once more after the last ray is gone, so it stays within `count` and
// a few hundred whatever the rays' numbers are.  `base`: its value before the
// warp asked for `want` rays.  Whether the block has no ray left after that:
SLRGPU_HD bool raysDrained(uint32_t base, uint32_t want, uint32_t count) { return base >= count || count - base <= want; }

}  // namespace slrgpu
