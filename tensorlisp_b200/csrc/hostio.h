// Host <-> device traffic of the C ABI: pinned memory that is kept between calls, staged copies of pageable memory
// that several host threads fill, and the two small kernels that move a program's small inputs and results
// between pinned host memory and the device inside the program's own launch sequence.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>

namespace tlb {

// ---- pinned host memory. Blocks are kept for reuse up to a bound (HOST_CACHE_LIMIT); what is handed out at any time
// is bounded too (HOST_LIVE_LIMIT): beyond it, and when pinning fails, pinned_alloc returns null and the caller uses
// pageable memory. Safe to use from several threads.
// PIN_RESULT: a fresh block only while the blocks of its size come back (a caller that keeps its results gets null).
// PIN_LIBRARY: a block the library itself cannot do without, whatever is handed out.
enum PinFor { PIN_CALLER, PIN_RESULT, PIN_LIBRARY };
void *pinned_alloc(uint64_t bytes, PinFor what);
// Makes no CUDA call (it runs wherever an array goes away): what the cache cannot hold is unpinned by the next pinned_alloc or
// pinned_trim.
void pinned_free(void *p);
void pinned_trim();
void pinned_device(int ordinal);                   // the device that pinning is done for
bool pinned_owns(const void *p, uint64_t bytes);   // [p, p + bytes) lies in a block that is handed out

// ---- host threads: runs fn(0) .. fn(n - 1), on the calling thread and up to `threads` - 1 others. When another caller
// has the helpers, everything runs on the calling thread.
void host_parallel(int n, int threads, const std::function<void(int)> &fn);

// ---- copies between caller memory (pageable or pinned) and the device on `st`.
// h2d: when it returns, the source has been read (the copy itself may still be on its way, in stream order).
// d2h: when it returns, the destination holds the data (everything in front of it on the stream has finished).
cudaError_t copy_h2d(int ordinal, void *dst, const void *src, uint64_t n, cudaStream_t st);
cudaError_t copy_d2h(int ordinal, void *dst, const void *src, uint64_t n, cudaStream_t st);

// ---- a program's pinned page
constexpr int IO_MAX_IN = 32, IO_MAX_OUT = 8;          // entries of the two tables
// An input of at most IO_IN_MAX bytes waits in the page. set_input and run of a program with one input in us, as a copy of its own / through the
// page: 128 KB 38.8 / 32.0, 192 KB 41.8 / 35.6, 256 KB 43.9 / 37.3, 384 KB 53.1 / 49.3, 512 KB 52.1 / 62.6, 1 MB 74 / 103.
constexpr uint64_t IO_IN_MAX = 256 << 10, IO_IN_TOTAL = 512 << 10;
constexpr uint64_t IO_OUT_SMALL = 64 << 10, IO_OUT_TOTAL = 64 << 10;    // a result of at most IO_OUT_SMALL goes there,
constexpr uint64_t IO_OUT_MAX = 2 << 20;                                // one of at most this into a pinned block of its own (4 MB: no gain)
struct IoPiece {
    uint64_t dev_off;    // byte offset in the program's io buffer (inputs) or arena (outputs), a multiple of 16
    uint64_t host;       // address in pinned memory, a multiple of 16
    uint64_t n16;        // 16-byte pieces
    uint64_t pad;
};
struct IoPage {
    int err;             // error word of the program's kernels (bounded waits, indices out of range)
    int pad0[15];
    int n_in, n_out, pad1[14];
    IoPiece in[IO_MAX_IN];
    IoPiece out[IO_MAX_OUT];
};
// In device memory, zero at first: CTAs of a fetch that have read the table, and the table of results that it found.
struct IoSync {
    uint32_t in_done;
    int n_out, pad[6];
    IoPiece out[IO_MAX_OUT];
};
// moves the n_in listed inputs from the page to the io buffer and sets n_in to 0 (bytes: what they may come to); takes over the
// table of results
cudaError_t launch_fetch_inputs(IoPage *page, void *io, IoSync *sync, uint64_t bytes, cudaStream_t st);
// moves the listed outputs from the arena to pinned memory, as the fetch in front of it in the sequence found them listed
cudaError_t launch_push_outputs(const void *arena, const IoSync *sync, uint64_t bytes, cudaStream_t st);

}  // namespace tlb
