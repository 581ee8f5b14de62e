#include "bounce_counts.h"

#include <sched.h>

#include <cstring>
#include <string>

#include "../../include/slrgpu.h"

namespace slrgpu {

void setError(const std::string &msg);

bool BounceCounts::wanted() {
    unsigned int flags = 0;
    return cudaGetDeviceFlags(&flags) != cudaSuccess || (flags & cudaDeviceScheduleMask) != cudaDeviceScheduleBlockingSync;
}

int BounceCounts::begin(uint32_t bounces, cudaStream_t stream) {
    if (bounces > capacity) {
        // a wave that ended in an error may have left kernels that still write
        if (host) cudaStreamSynchronize(stream);
        release();
        const cudaError_t e = cudaMallocHost((void**)&host, bounces * sizeof(*host));
        if (e != cudaSuccess) {
            host = nullptr;
            setError(std::string("bounce counts: ") + cudaGetErrorString(e));
            return SLRGPU_ERR_OUT_OF_MEMORY;
        }
        capacity = bounces;
        std::memset(host, 0, bounces * sizeof(*host));
        tag = 0;
    }
    ++tag;   // the waves of 2^32 before it are long complete
    if (tag == 0) tag = 1;
    return SLRGPU_OK;
}

cudaError_t BounceCounts::get(uint32_t bounce, cudaStream_t stream, uint32_t* count) {
    const volatile unsigned long long* word = host + bounce;
    // as cudaStreamSynchronize would wait
    unsigned int flags = 0;
    const bool yield = cudaGetDeviceFlags(&flags) == cudaSuccess &&
                       (flags & cudaDeviceScheduleMask) == cudaDeviceScheduleYield;
    for (uint32_t looks = 1;; ++looks) {
        unsigned long long v = *word;
        if ((uint32_t)(v >> 32) == tag) {
            *count = (uint32_t)v;
            return cudaSuccess;
        }
        if (!yield && (looks & 0xfff) != 0) continue;
        // a kernel of the wave that was refused at its launch never writes
        const cudaError_t pending = cudaGetLastError();
        if (pending != cudaSuccess && pending != cudaErrorNotReady) return pending;
        // a stream that has run dry has written the word, or failed
        const cudaError_t e = cudaStreamQuery(stream);
        if (e != cudaSuccess) cudaGetLastError();   // "not ready" is no error: no trace for the check after the wave
        if (e == cudaErrorNotReady) {
            if (yield) sched_yield();
            continue;
        }
        v = *word;
        *count = (uint32_t)v;
        if (e != cudaSuccess) return e;
        return (uint32_t)(v >> 32) == tag ? cudaSuccess : cudaErrorUnknown;
    }
}

void BounceCounts::release() {
    if (host) cudaFreeHost(host);
    host = nullptr;
    capacity = 0;
}

}  // namespace slrgpu
