// Pinned memory pool, staged host copies and the in-stream input / output kernels (hostio.h).
//
// What bounds a host copy here: a pageable cudaMemcpy goes through the driver's own staging on one thread (measured on
// the B200 host: 443 us for 8 MB, 19 GB/s, and a fresh result array pays a page fault per 4 KB on top), and every
// blocking copy ends with a stream synchronisation of 8 to 10 us however small it is. So large copies are staged by
// several host threads into a pinned ring while the earlier chunks are on the link, results are read straight into
// pinned arrays, and inputs of at most 256 KB and results of at most 2 MB make no copy call at all: a kernel at the head of
// the program's launch sequence reads them over the link from a pinned page, one at its tail writes them into pinned memory that the
// caller then takes over.
#include <emmintrin.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "hostio.h"
#include "pdl.cuh"

namespace tlb {

// ---------------------------------------------------------------------------- pinned pool
namespace {

constexpr uint64_t HOST_CACHE_LIMIT = 256ull << 20;   // bytes kept for reuse
constexpr uint64_t HOST_LIVE_LIMIT = 1024ull << 20;   // bytes handed out at any time
// Fresh result blocks per size: two (the caller lets go of one result when it has the next), and one more for every eight times that
// a block was used again. Pinning is slow: a call whose result went into a fresh block took 0.6 to 2.5 ms at 1 MB and 6.5 to 9 ms at
// 16 MB, into ordinary memory 0.45 and 2 to 3.5 ms (most of it the first touch of its pages), into a block that came back 0.06 and
// 0.39 ms. A caller that keeps its results would pay for a fresh block every time.
constexpr uint64_t RESULT_FRESH = 2, RESULT_HITS = 8;

struct PinnedPool {
    std::mutex m;
    std::map<uintptr_t, uint64_t> live;                    // handed out: address -> block size
    std::multimap<uint64_t, void *> idle;                  // by block size
    uint64_t live_bytes = 0, idle_bytes = 0;
    struct Use { uint64_t fresh = 0, hits = 0; };
    std::map<uint64_t, Use> results;                       // by block size
    std::atomic<int> device{0};
};
// never destroyed: blocks may be given back while the process ends
PinnedPool &pool() {
    static PinnedPool *p = new PinnedPool;
    return *p;
}
// block sizes: powers of two and their halfway points, 64 KB at least
uint64_t block_size(uint64_t bytes) {
    uint64_t b = 64 << 10;
    while (b < bytes) {
        if (b + b / 2 >= bytes) return b + b / 2;
        b *= 2;
    }
    return b;
}

}  // namespace

void pinned_device(int ordinal) { pool().device = ordinal; }

void pinned_trim() {
    PinnedPool &p = pool();
    std::vector<void *> drop;
    {
        std::lock_guard<std::mutex> lock(p.m);
        while (p.idle_bytes > HOST_CACHE_LIMIT) {   // the largest go first
            auto last = std::prev(p.idle.end());
            p.idle_bytes -= last->first;
            drop.push_back(last->second);
            p.idle.erase(last);
        }
    }
    if (!drop.empty()) cudaSetDevice(p.device);
    for (void *d : drop) cudaFreeHost(d);
}

void *pinned_alloc(uint64_t bytes, PinFor what) {
    const uint64_t b = block_size(bytes);
    PinnedPool &p = pool();
    pinned_trim();
    {
        std::lock_guard<std::mutex> lock(p.m);
        if (what != PIN_LIBRARY && p.live_bytes + b > HOST_LIVE_LIMIT) return nullptr;
        auto it = p.idle.find(b);
        if (what == PIN_RESULT) {
            PinnedPool::Use &use = p.results[b];
            if (it != p.idle.end()) use.hits++;
            else if (use.fresh >= RESULT_FRESH + use.hits / RESULT_HITS) return nullptr;
            else use.fresh++;
        }
        if (it != p.idle.end()) {
            void *q = it->second;
            p.idle.erase(it);
            p.idle_bytes -= b;
            p.live[(uintptr_t)q] = b;
            p.live_bytes += b;
            return q;
        }
    }
    void *q = nullptr;
    if (what != PIN_LIBRARY) cudaSetDevice(p.device);   // (the library's own calls have set theirs)
    if (cudaHostAlloc(&q, b, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(p.m);
    p.live[(uintptr_t)q] = b;
    p.live_bytes += b;
    return q;
}

void pinned_free(void *q) {
    if (!q) return;
    PinnedPool &p = pool();
    std::lock_guard<std::mutex> lock(p.m);
    auto it = p.live.find((uintptr_t)q);
    if (it == p.live.end()) return;
    const uint64_t b = it->second;
    p.live.erase(it);
    p.live_bytes -= b;
    p.idle.emplace(b, q);
    p.idle_bytes += b;
}

bool pinned_owns(const void *q, uint64_t bytes) {
    PinnedPool &p = pool();
    std::lock_guard<std::mutex> lock(p.m);
    auto it = p.live.upper_bound((uintptr_t)q);
    if (it == p.live.begin()) return false;
    --it;
    const uint64_t at = (uintptr_t)q - it->first;
    return at <= it->second && bytes <= it->second - at;
}

// ---------------------------------------------------------------------------- host threads
namespace {

struct Helpers {
    std::mutex busy;                 // one parallel region at a time
    std::mutex m;
    std::condition_variable wake;
    std::vector<std::thread> threads;
    const std::function<void(int)> *fn = nullptr;
    std::atomic<int> next{0}, left{0};
    int n = 0, want = 0, inside = 0;
    uint64_t generation = 0;

    void work(const std::function<void(int)> &f, int count) {
        for (int i; (i = next.fetch_add(1)) < count;) {
            f(i);
            left.fetch_sub(1, std::memory_order_release);
        }
    }
    void loop() {
        uint64_t seen = 0;
        std::unique_lock<std::mutex> lock(m);
        for (;;) {
            wake.wait(lock, [&] { return generation != seen; });
            seen = generation;
            if (want <= 0 || !fn) continue;
            want--;
            inside++;
            const auto *f = fn;
            const int count = n;
            lock.unlock();
            work(*f, count);
            lock.lock();
            inside--;
        }
    }
};
Helpers &helpers() {
    static Helpers *h = new Helpers;   // never destroyed: its threads sleep until the process ends
    return *h;
}
int helper_limit() {
    static const int n = std::max(1, std::min(8, (int)std::thread::hardware_concurrency() / 2));
    return n;
}

}  // namespace

void host_parallel(int n, int threads, const std::function<void(int)> &fn) {
    Helpers &h = helpers();
    threads = std::min({threads, n, helper_limit()});
    std::unique_lock<std::mutex> busy(h.busy, std::defer_lock);
    if (threads <= 1 || !busy.try_lock()) {
        for (int i = 0; i < n; i++) fn(i);
        return;
    }
    {
        std::lock_guard<std::mutex> lock(h.m);
        while ((int)h.threads.size() < threads - 1) {
            try {
                h.threads.emplace_back([&h] { h.loop(); });
                h.threads.back().detach();
            } catch (...) {
                break;   // fewer helpers
            }
        }
        h.fn = &fn;
        h.n = n;
        h.next = 0;
        h.left = n;
        h.want = threads - 1;
        h.generation++;
    }
    h.wake.notify_all();
    h.work(fn, n);
    while (h.left.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    // no helper may still hold a pointer to fn
    for (;;) {
        std::lock_guard<std::mutex> lock(h.m);
        h.fn = nullptr;
        h.want = 0;
        if (h.inside == 0) break;
    }
}

// ---------------------------------------------------------------------------- staged copies
namespace {

constexpr int RING_SLOTS = 16;
constexpr uint64_t RING_CHUNK = 1 << 20;
// Bytes per chunk and threads for a copy of n bytes: a chunk costs about 5 us of driver calls, and the link idles
// until the first one is staged.
uint64_t chunk_of(uint64_t n) { return n >= (16 << 20) ? RING_CHUNK : (n >= (2 << 20) ? 512 << 10 : 256 << 10); }
int threads_of(uint64_t n) { return n >= (2 << 20) ? 4 : (n >= (512 << 10) ? 2 : 1); }

// memcpy with stores that bypass the caches (x86-64 baseline instructions)
void stream_copy(char *d, const char *s, uint64_t n) {
    const uint64_t head = std::min<uint64_t>(n, (16 - ((uintptr_t)d & 15)) & 15);
    std::memcpy(d, s, head);
    d += head;
    s += head;
    n -= head;
    uint64_t i = 0;
    for (; i + 64 <= n; i += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i *)(s + i)), b = _mm_loadu_si128((const __m128i *)(s + i + 16)),
                      c = _mm_loadu_si128((const __m128i *)(s + i + 32)), e = _mm_loadu_si128((const __m128i *)(s + i + 48));
        _mm_stream_si128((__m128i *)(d + i), a);
        _mm_stream_si128((__m128i *)(d + i + 16), b);
        _mm_stream_si128((__m128i *)(d + i + 32), c);
        _mm_stream_si128((__m128i *)(d + i + 48), e);
    }
    std::memcpy(d + i, s + i, n - i);
    _mm_sfence();
}

// One ring per device: chunk k of a copy goes through slot k mod RING_SLOTS; a slot's event tells when the link has
// read (or written) it.
struct Ring {
    std::mutex m;                      // one staged copy at a time
    char *mem = nullptr;
    cudaEvent_t ev[RING_SLOTS] = {};
    std::atomic<uint64_t> issued[RING_SLOTS];   // 1 + number of the last chunk whose copy has been enqueued through the slot
    uint64_t next = 0;                 // chunks so far
    bool ok = false;
};
Ring &ring(int ordinal) {
    static Ring *r = new Ring[64];
    return r[ordinal & 63];
}
bool ring_ready(Ring &r) {
    if (r.ok) return true;
    if (!r.mem) r.mem = (char *)pinned_alloc(RING_SLOTS * RING_CHUNK, PIN_LIBRARY);
    if (!r.mem) return false;
    for (int s = 0; s < RING_SLOTS; s++) {
        r.issued[s] = 0;
        if (!r.ev[s] && cudaEventCreateWithFlags(&r.ev[s], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    }
    return r.ok = true;
}
// memory the driver already knows as pinned: ours, or the caller's
bool is_pinned(const void *p, uint64_t n) {
    if (pinned_owns(p, n)) return true;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged;
}

}  // namespace

cudaError_t copy_h2d(int ordinal, void *dst, const void *src, uint64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    Ring &r = ring(ordinal);
    if (is_pinned(src, n)) {
        cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    std::lock_guard<std::mutex> lock(r.m);
    if (!ring_ready(r)) {
        cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    const uint64_t chunk = chunk_of(n);
    const int chunks = (int)((n + chunk - 1) / chunk);
    const uint64_t base = r.next;
    std::atomic<int> err{cudaSuccess};
    host_parallel(chunks, threads_of(n), [&](int c) {
        cudaError_t e = cudaSetDevice(ordinal);   // a helper thread begins with device 0
        if (e != cudaSuccess) err = e;
        const uint64_t k = base + c;
        const int s = (int)(k % RING_SLOTS);
        if (k >= RING_SLOTS) {   // the chunk that used the slot before: enqueued (perhaps by another thread), then read by the link
            while (r.issued[s].load(std::memory_order_acquire) < k - RING_SLOTS + 1) std::this_thread::yield();
            e = cudaEventSynchronize(r.ev[s]);
            if (e != cudaSuccess) err = e;
        }
        const uint64_t off = (uint64_t)c * chunk, m = std::min(chunk, n - off);
        char *slot = r.mem + s * RING_CHUNK;
        stream_copy(slot, (const char *)src + off, m);
        e = cudaMemcpyAsync((char *)dst + off, slot, m, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(r.ev[s], st);
        if (e != cudaSuccess) err = e;
        r.issued[s].store(k + 1, std::memory_order_release);
    });
    r.next = base + chunks;
    return (cudaError_t)err.load();
}

cudaError_t copy_d2h(int ordinal, void *dst, const void *src, uint64_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    Ring &r = ring(ordinal);
    std::unique_lock<std::mutex> lock(r.m, std::defer_lock);
    bool staged = n >= (128 << 10) && !is_pinned(dst, n);
    if (staged) {
        lock.lock();
        staged = ring_ready(r);
    }
    if (!staged) {
        cudaError_t e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    const uint64_t chunk = chunk_of(n);
    const int chunks = (int)((n + chunk - 1) / chunk);
    const uint64_t base = r.next;
    for (int s = 0; s < RING_SLOTS; s++)   // uploads that still wait in the ring
        if (r.issued[s].load() > 0) {
            const cudaError_t e = cudaEventSynchronize(r.ev[s]);
            if (e != cudaSuccess) return e;
        }
    std::atomic<int> err{cudaSuccess};
    // half the ring is on the link while the other half is copied out
    const int wave = RING_SLOTS / 2;
    auto issue = [&](int w) {
        r.next = base + std::min(chunks, (w + 1) * wave);   // behind an error no further wave is sent: the numbers of its chunks stay free
        for (int c = w * wave; c < std::min(chunks, (w + 1) * wave); c++) {
            const uint64_t k = base + c;
            const int s = (int)(k % RING_SLOTS);
            const uint64_t off = (uint64_t)c * chunk, m = std::min(chunk, n - off);
            cudaError_t e = cudaMemcpyAsync(r.mem + s * RING_CHUNK, (const char *)src + off, m, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(r.ev[s], st);
            if (e != cudaSuccess) err = e;
            r.issued[s].store(k + 1, std::memory_order_release);
        }
    };
    const int waves = (chunks + wave - 1) / wave;
    issue(0);
    for (int w = 0; w < waves && err == cudaSuccess; w++) {
        if (w + 1 < waves) issue(w + 1);
        const int c0 = w * wave, c1 = std::min(chunks, (w + 1) * wave);
        host_parallel(c1 - c0, threads_of(n), [&](int i) {
            const int c = c0 + i, s = (int)((base + c) % RING_SLOTS);
            cudaError_t e = cudaSetDevice(ordinal);
            if (e == cudaSuccess) e = cudaEventSynchronize(r.ev[s]);
            if (e != cudaSuccess) {
                err = e;
                return;
            }
            const uint64_t off = (uint64_t)c * chunk;
            stream_copy((char *)dst + off, r.mem + s * RING_CHUNK, std::min(chunk, n - off));
        });
    }
    const cudaError_t e = cudaStreamSynchronize(st);   // also behind an error: nothing writes the ring any more
    return err != cudaSuccess ? (cudaError_t)err.load() : e;
}

// ---------------------------------------------------------------------------- the page kernels
namespace {

__device__ __forceinline__ uint4 ld_host(const void *p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// What these cost is round trips over the link (the table, then the data: about 1.5 us each) and reads by many CTAs: those of
// pinned memory queue up, 1.6 us for every CTA that reads the table. So few CTAs fetch, and the first of them leaves the table of the
// results in device memory, where the CTAs of the second kernel find it: 8 KB each, 1 MB of results in 24 us (one CTA wrote 10 GB/s). The
// fetch does not let its successors start early: beside its CTA a product's came to lie two to an SM (a [32000 x 4096] Q6_K product with its
// inputs and results 57 -> 76 us, the feed-forward block of one token 43 -> 51).
__global__ void __launch_bounds__(1024) k_io_fetch(IoPage *page, char *dev, IoSync *sync) {
    __shared__ uint4 ent[IO_MAX_IN][2];
    __shared__ int s_n;
    __shared__ uint32_t first[IO_MAX_IN + 1];
    const int tid = threadIdx.x;
    if (tid < 2 * IO_MAX_IN) ent[tid >> 1][tid & 1] = ld_host(reinterpret_cast<const uint4 *>(page->in) + tid);
    if (tid == 2 * IO_MAX_IN) {
        const int n = *(volatile int *)&page->n_in;
        s_n = n < 0 ? 0 : (n > IO_MAX_IN ? IO_MAX_IN : n);
    }
    if (blockIdx.x == 0 && tid >= 128) {
        const int i = tid - 128;
        if (i < 2 * IO_MAX_OUT) reinterpret_cast<uint4 *>(sync->out)[i] = ld_host(reinterpret_cast<const uint4 *>(page->out) + i);
        if (i == 2 * IO_MAX_OUT) sync->n_out = *(volatile int *)&page->n_out;
    }
    __syncthreads();
    const int n = s_n;
    if (tid == 0) {
        uint32_t at = 0;
        for (int i = 0; i < n; i++) {
            first[i] = at;
            at += ent[i][1].x;
        }
        first[n] = at;
        if (gridDim.x == 1 || atomicAdd(&sync->in_done, 1u) == gridDim.x - 1) {   // every CTA has read the table
            sync->in_done = 0;
            *(volatile int *)&page->n_in = 0;
        }
    }
    __syncthreads();
    const uint32_t total = first[n];
    for (uint32_t i0 = blockIdx.x * 4096 + tid; i0 < total; i0 += gridDim.x * 4096) {
        uint4 v[4];
        char *to[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t i = i0 + u * 1024;
            to[u] = nullptr;
            if (i >= total) continue;
            int e = 0;
            while (i >= first[e + 1]) e++;
            to[u] = dev + ((uint64_t)ent[e][0].x | ((uint64_t)ent[e][0].y << 32)) + (uint64_t)(i - first[e]) * 16;
            v[u] = ld_host(reinterpret_cast<const char *>((uint64_t)ent[e][0].z | ((uint64_t)ent[e][0].w << 32)) + (uint64_t)(i - first[e]) * 16);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (to[u]) *reinterpret_cast<uint4 *>(to[u]) = v[u];
    }
}
__global__ void __launch_bounds__(512) k_io_push(const char *dev, const IoSync *sync) {
    griddep_wait();
    const int n = min(max(sync->n_out, 0), IO_MAX_OUT);
    for (int e = 0; e < n; e++) {
        const IoPiece p = sync->out[e];
        const uint4 *from = reinterpret_cast<const uint4 *>(dev + p.dev_off);
        uint4 *to = reinterpret_cast<uint4 *>(p.host);
#pragma unroll 2
        for (uint64_t i = blockIdx.x * 512 + threadIdx.x; i < p.n16; i += gridDim.x * 512) to[i] = from[i];
    }
}

}  // namespace

static_assert(sizeof(IoPiece) == 32, "an entry is two 16-byte loads");

cudaError_t launch_fetch_inputs(IoPage *page, void *io, IoSync *sync, uint64_t bytes, cudaStream_t st) {
    k_io_fetch<<<bytes > (64 << 10) ? 4 : 1, 1024, 0, st>>>(page, (char *)io, sync);
    return cudaGetLastError();
}
cudaError_t launch_push_outputs(const void *arena, const IoSync *sync, uint64_t bytes, cudaStream_t st) {
    return launch_pdl(k_io_push, dim3((unsigned)std::max<uint64_t>(1, std::min<uint64_t>(64, (bytes + (8 << 10) - 1) / (8 << 10)))), dim3(512), 0, st, (const char *)arena, sync);
}

}  // namespace tlb
