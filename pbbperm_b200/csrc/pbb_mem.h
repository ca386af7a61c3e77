// Device memory and streams of the library's objects and calls.
//
// An engine, a pool or a bound call needs its buffers for milliseconds, and
// cudaMalloc / cudaFree take as long as a small search (creating and
// destroying a 12x10 engine: 3.2 ms of a 4.2 ms solve, and tens of
// milliseconds on a busy host).  Buffers are therefore kept, per device: those
// up to PBB_BIG_BLOCK in a stream-ordered pool that holds on to at most
// PBB_POOL_KEEP bytes of freed memory, larger ones -- a pool grows by them ten
// times slower than cudaMalloc does (1.6 GB: 40 ms and 3) -- in a list of freed
// blocks of at most PBB_BIG_KEEP bytes.  More than that goes back to the driver
// as it is freed, and all of it before an allocation fails.  Streams are kept
// too, a few per device.  All of it is safe from any thread.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#define PBB_BIG_BLOCK (256ull << 20)
#define PBB_POOL_KEEP (1ull << 30)
#define PBB_BIG_KEEP (2ull << 30)
#define PBB_STREAMS_KEPT 8

namespace pbbh {
// `device` is the current device; the memory belongs to stream `st`'s order
cudaError_t mem_alloc(void** out, size_t bytes, int device, cudaStream_t st);
// the work that used p has finished
void mem_free(void* p, cudaStream_t st);
// a non-blocking stream of the current device
cudaError_t stream_take(cudaStream_t* st, int device);
// `st` has no work left
void stream_give(cudaStream_t st, int device);

// sub-buffers of one block, each on a 256-byte boundary
struct Carver {
    size_t bytes = 0;
    size_t take(size_t n)
    {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    }
};
}  // namespace pbbh
