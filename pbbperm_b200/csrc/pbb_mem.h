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
// as it is freed, and all of it before an allocation fails or when the caller
// asks for it (pbb_release_memory).  Streams are kept too, a few per device.
// All of it is safe from any thread.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#define PBB_BIG_BLOCK (256ull << 20)
#define PBB_POOL_KEEP (1ull << 30)
#define PBB_BIG_KEEP (2ull << 30)
#define PBB_STREAMS_KEPT 8

namespace pbbh {
// A stream lent to an object or call.  The object's memory, events and graphs
// are of the same context; they die with it when the device is reset.
struct Lease {
    cudaStream_t st = nullptr;
    int device = 0;
    unsigned long long context = 0;
};
// All of these: the lease's device is current.
// a non-blocking stream
cudaError_t stream_take(Lease* l, int device);
// the context of the lease is the device's current one: its handles are valid
bool alive(const Lease& l);
// memory in the order of the lease's stream
cudaError_t mem_alloc(void** out, size_t bytes, const Lease& l);
// the work that used p has finished; nothing to do when the lease is not alive
void mem_free(void* p, const Lease& l);
// the stream has no work left but frees; forgotten when the lease is not alive
void stream_give(Lease& l);
// what is kept of the current device goes back to the driver
void mem_release(int device);

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
