/* Walks the rays of ray-query kernels as their warps do (ray_blocks.h): every
 * block's eight warps ask for 1 to 32 rays in turn until each has seen the
 * block drained.  Every ray of every walked block is taken once, no other one
 * is, and a warp asks a bounded number of times, up to the largest n. */
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../slr_gb300/csrc/ray_blocks.h"

using namespace slrgpu;

static uint32_t rnd() {
    static uint64_t s = 88172645463325252ull;
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    return (uint32_t)(s >> 32);
}

static bool walk(uint32_t n, uint32_t blocks, uint32_t block) {
    const RayBlock own = rayBlock(n, blocks, block);
    std::vector<uint8_t> taken(own.count, 0);
    uint32_t cursor = 0;
    bool drained[8] = {};
    uint64_t asks = 0;
    for (int left = 8; left > 0;) {
        const int w = (int)(rnd() & 7);
        if (drained[w]) continue;
        if (++asks > (uint64_t)own.count + 8) return false;   // must end
        const uint32_t want = 1 + (rnd() & 31), base = cursor;
        cursor += want;
        if (cursor < base) return false;                      // wrapped
        drained[w] = raysDrained(base, want, own.count);
        left -= drained[w];
        for (uint32_t r = 0; r < want; ++r) {
            if (base + r >= own.count) continue;
            const uint32_t i = own.first + (base + r);
            if (i < own.first || i >= n || taken[base + r]++) return false;
        }
    }
    for (uint8_t t : taken)
        if (t != 1) return false;
    return true;
}

int main() {
    const uint32_t ns[] = {1, 2, 255, 256, 257, 1000003, 1u << 22, 0x7fffffffu, 0xffffff00u, 0xfffffff0u, 0xffffffffu};
    const uint32_t grids[] = {1, 152, 608, 1216};
    int bad = 0, walks = 0;
    for (uint32_t n : ns)
        for (uint32_t blocks : grids) {
            if (n / blocks > (1u << 26)) continue;            // no such launch: a grid fills the GPU
            uint64_t sum = 0;
            for (uint32_t b = 0; b < blocks; ++b) {
                const RayBlock r = rayBlock(n, blocks, b);
                if (r.count && r.first != sum) ++bad;         // consecutive ranges
                sum += r.count;
            }
            if (sum != n) ++bad;
            const uint32_t some[] = {0, blocks / 2, blocks - 1, (uint32_t)((n - 1) / raysPerBlock(n, blocks))};
            for (uint32_t b : some) {
                ++walks;
                if (!walk(n, blocks, b)) {
                    std::printf("n %u blocks %u block %u\n", n, blocks, b);
                    ++bad;
                }
            }
        }
    std::printf("walks %d bad %d\n", walks, bad);
    return bad != 0;
}
