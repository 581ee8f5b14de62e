/* The host's wait for a wave's bounce counts (bounce_counts.cpp) against a CUDA
 * runtime made of the few calls it needs, whose answers each case scripts. */
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <string>
#include <vector>

#include "../slr_gb300/csrc/bounce_counts.h"

static cudaError_t g_last = cudaSuccess;          // the thread's pending error
static std::function<cudaError_t()> g_query;      // the stream's state
static unsigned int g_flags = 0;
static int g_queries = 0;
static std::vector<std::string> g_calls;

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { g_calls.push_back("free"); std::free(p); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { g_calls.push_back("synchronize"); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetDeviceFlags(unsigned int* f) { *f = g_flags; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaStreamQuery(cudaStream_t) {
    ++g_queries;
    const cudaError_t e = g_query();
    if (e != cudaSuccess) g_last = e;             // as the runtime records it
    return e;
}
}
namespace slrgpu { void setError(const std::string &) {} }

static int g_bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); ++g_bad; } } while (0)

int main() {
    using slrgpu::BounceCounts;
    BounceCounts c;
    uint32_t n = 0;
    auto word = [&](uint32_t tag, uint32_t paths) { return (unsigned long long)tag << 32 | paths; };
    auto fresh = [&]() { g_last = cudaSuccess; g_queries = 0; n = 0; CHECK(c.begin(8, nullptr) == 0); };

    fresh();                                      // the word is there
    c.host[3] = word(c.tag, 77);
    CHECK(c.get(3, nullptr, &n) == cudaSuccess && n == 77 && g_queries == 0);

    fresh();                                      // the last wave's word is not this wave's
    g_query = [&]() { if (g_queries == 3) c.host[3] = word(c.tag, 5); return cudaErrorNotReady; };
    CHECK(c.get(3, nullptr, &n) == cudaSuccess && n == 5 && g_queries == 3);
    CHECK(g_last == cudaSuccess);                 // a running stream leaves no error behind

    fresh();                                      // a kernel was refused at its launch: its error, once
    g_last = cudaErrorLaunchOutOfResources;
    g_query = [&]() { return g_queries < 2 ? cudaErrorNotReady : cudaSuccess; };
    CHECK(c.get(2, nullptr, &n) == cudaErrorLaunchOutOfResources);
    CHECK(g_last == cudaSuccess);

    fresh();                                      // the stream has run dry without the word
    g_query = [&]() { return cudaSuccess; };
    CHECK(c.get(2, nullptr, &n) == cudaErrorUnknown && g_last == cudaSuccess);

    fresh();                                      // ... or wrote it between the two looks
    g_query = [&]() { c.host[2] = word(c.tag, 9); return cudaSuccess; };
    CHECK(c.get(2, nullptr, &n) == cudaSuccess && n == 9);

    fresh();                                      // the stream failed
    g_query = [&]() { return cudaErrorIllegalAddress; };
    CHECK(c.get(2, nullptr, &n) == cudaErrorIllegalAddress && g_last == cudaSuccess);

    c.tag = 0xffffffffu;                          // tag 0 marks no wave
    fresh();
    CHECK(c.tag == 1);

    g_calls.clear();                              // more bounces: nothing writes to the old words any more
    CHECK(c.begin(20, nullptr) == 0 && c.capacity == 20);
    CHECK((g_calls == std::vector<std::string>{"synchronize", "free"}));

    // Where waiting threads are set to sleep the host does not look; where they yield it looks every time.
    for (unsigned int flags : {0u, (unsigned int)cudaDeviceScheduleSpin, (unsigned int)cudaDeviceScheduleYield}) {
        g_flags = flags | cudaDeviceMapHost;
        CHECK(BounceCounts::wanted());
        fresh();
        g_query = [&]() { if (g_queries == 3) c.host[2] = word(c.tag, 4); return cudaErrorNotReady; };
        CHECK(c.get(2, nullptr, &n) == cudaSuccess && n == 4 && g_queries == 3 && g_last == cudaSuccess);
    }
    g_flags = cudaDeviceScheduleBlockingSync | cudaDeviceMapHost;
    CHECK(!BounceCounts::wanted());
    c.release();
    std::printf("bad %d\n", g_bad);
    return g_bad != 0;
}
