// The number of paths that start each bounce of a wave, as the host sees it
// while the wave runs.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdint>

namespace slrgpu {

// The bounce's first kernel writes a word of pinned host memory: the wave's
// tag in the high half, the bounce's paths in the low one.
struct BounceCounts {
    unsigned long long* host = nullptr;   // [capacity], pinned
    uint32_t capacity = 0;
    uint32_t tag = 0;

    // Whether the host looks at all: it would wait awake, so not where the
    // device's waiting threads are set to sleep (cudaDeviceScheduleBlockingSync).
    static bool wanted();
    // A new wave on the stream.  On failure, an error code of the C ABI.
    int begin(uint32_t bounces, cudaStream_t stream);
    // Waits until the bounce has started.  An error that is pending when the
    // wait looks (a kernel that was refused at its launch), or an error of
    // the stream, ends the wait, is returned, and is pending no longer.
    cudaError_t get(uint32_t bounce, cudaStream_t stream, uint32_t* count);
    void release();
};

}  // namespace slrgpu
