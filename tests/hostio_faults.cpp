// The staged copies of csrc/hostio.cu against a CUDA runtime that fails on demand: the linker sends the calls below here
// (--wrap), device memory is ordinary memory, and copies happen at once. One scenario per run, named on the command line;
// exit code 0 means that it held.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "hostio.h"

namespace {
constexpr int ORDINAL = 3;
std::atomic<int> copies{0}, waits{0}, fail_copy{-1}, fail_wait{-1}, stray{0}, pinned{0}, unpinned{0};
thread_local int device = 0;
void on_device() {
    if (device != ORDINAL) stray++;
}
}  // namespace

extern "C" {
cudaError_t __wrap_cudaSetDevice(int d) {
    device = d;
    return cudaSuccess;
}
cudaError_t __wrap_cudaHostAlloc(void **p, size_t n, unsigned) {
    on_device();
    pinned++;
    *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t __wrap_cudaFreeHost(void *p) {
    on_device();
    unpinned++;
    std::free(p);
    return cudaSuccess;
}
cudaError_t __wrap_cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t __wrap_cudaGetLastError() { return cudaSuccess; }
cudaError_t __wrap_cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = (cudaEvent_t)1;
    return cudaSuccess;
}
cudaError_t __wrap_cudaEventRecord(cudaEvent_t, cudaStream_t) {
    on_device();
    return cudaSuccess;
}
cudaError_t __wrap_cudaEventSynchronize(cudaEvent_t) {
    on_device();
    return waits++ == fail_wait ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t __wrap_cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    on_device();
    if (copies++ == fail_copy) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t __wrap_cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}

#define HOLDS(x)                                      \
    do {                                              \
        if (!(x)) {                                   \
            std::printf("does not hold: %s\n", #x);   \
            return 1;                                 \
        }                                             \
    } while (0)

// Results that are kept do not pin a block each; those that are let go of are used again, several a step too; freeing makes no CUDA
// call, and what the cache cannot hold goes with the next request.
int results() {
    using namespace tlb;
    pinned_device(ORDINAL);
    std::vector<void *> kept;
    for (int i = 0; i < 50; i++) kept.push_back(pinned_alloc(500 << 10, PIN_RESULT));
    HOLDS(pinned <= 4);
    for (void *p : kept) pinned_free(p);
    for (int i = 0; i < 200; i++) {   // three blocks a step, the last step's still held
        std::vector<void *> now;
        for (int k = 0; k < 3; k++) now.push_back(pinned_alloc(500 << 10, PIN_RESULT));
        if (i > 100) HOLDS(now[0] && now[1] && now[2]);
        if (i > 0)
            for (void *p : kept) pinned_free(p);
        kept = now;
    }
    HOLDS(pinned <= 8);
    for (void *p : kept) pinned_free(p);
    const int before = pinned;
    std::vector<void *> own;          // what a caller asks for itself is not refused, up to 1 GB
    for (int i = 0; i < 6; i++) own.push_back(pinned_alloc(128 << 20, PIN_CALLER));
    for (void *p : own) HOLDS(p != nullptr);
    HOLDS(pinned == before + 6 && pinned_alloc(512 << 20, PIN_CALLER) == nullptr);
    for (void *p : own) pinned_free(p);
    HOLDS(unpinned == 0);             // no CUDA call where an array goes away
    pinned_trim();
    HOLDS(unpinned >= 4 && stray == 0);
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    const size_t n = (40u << 20) + 12345;   // 41 chunks, six half rings
    std::vector<char> host(n), dev(n), back(n);
    for (size_t i = 0; i < n; i++) host[i] = (char)(i * 2654435761u >> 13);
    if (what == "results") return results();
    cudaSetDevice(ORDINAL);
    auto up = [&] { return tlb::copy_h2d(ORDINAL, dev.data(), host.data(), n, nullptr); };
    auto down = [&] {
        std::memset(back.data(), 0, n);
        return tlb::copy_d2h(ORDINAL, back.data(), dev.data(), n, nullptr);
    };
    auto same = [&] { return std::memcmp(host.data(), dev.data(), n) == 0 && std::memcmp(host.data(), back.data(), n) == 0; };
    if (what == "device_up" || what == "device_down") {   // every call is made for the copy's device, on threads that begin with another one
        for (int i = 0; i < 20; i++) HOLDS((what == "device_up" ? up() : down()) == cudaSuccess);
        HOLDS(stray == 0);
        return 0;
    }
    HOLDS(up() == cudaSuccess && down() == cudaSuccess && same());
    // a failing call is reported, and the copies after it are whole again
    const int at = argc > 2 ? std::atoi(argv[2]) : 0;
    const bool upload = what == "h2d_copy" || what == "h2d_wait", copy = what == "h2d_copy" || what == "d2h_copy";
    (copy ? fail_copy : fail_wait) = (copy ? copies : waits) + at;
    HOLDS((upload ? up() : down()) == cudaErrorUnknown);
    fail_copy = fail_wait = -1;
    std::memset(dev.data(), 0, n);
    for (int i = 0; i < 3; i++) HOLDS(up() == cudaSuccess && down() == cudaSuccess && same());
    return 0;
}
