// Device memory and streams kept between objects (pbb_mem.h).
#include <mutex>
#include <unordered_map>
#include <vector>

#include "pbb_mem.h"

namespace {

#define PBB_MEM_DEVICES 64

std::mutex g_mem_mutex;
cudaMemPool_t g_pool[PBB_MEM_DEVICES];
bool g_pool_tried[PBB_MEM_DEVICES];
std::vector<cudaStream_t> g_streams[PBB_MEM_DEVICES];

struct BigBlock {
    void* p;
    size_t bytes;
    int device;
};
std::vector<BigBlock> g_kept;                          // free
std::unordered_map<void*, BigBlock> g_big;             // in use

// The current context's identity (a device that was reset gets a new one), 0
// where the driver does not say.
unsigned long long context_id()
{
    typedef int (*GetId)(void*, unsigned long long*);
    static const GetId get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        const bool ok = cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        cudaGetLastError();
        return ok ? reinterpret_cast<GetId>(f) : nullptr;
    }();
    unsigned long long id = 0;
    return get && get(nullptr, &id) == 0 ? id : 0;
}

// What is known of a device belongs to its context: with another one current,
// it is gone and forgotten, the blocks in use too.  What those are replaced by
// may stand at the same addresses, so their owners are told apart by the
// context of their lease, not by the address.
unsigned long long g_context[PBB_MEM_DEVICES];

unsigned long long check_context(int device)
{
    const unsigned long long id = context_id();
    if (device < 0 || device >= PBB_MEM_DEVICES) return id;
    std::lock_guard<std::mutex> lock(g_mem_mutex);
    if (g_context[device] == id) return id;
    g_context[device] = id;
    g_pool[device] = nullptr;
    g_pool_tried[device] = false;
    g_streams[device].clear();
    for (size_t i = 0; i < g_kept.size();) {
        if (g_kept[i].device == device) g_kept.erase(g_kept.begin() + i);
        else i++;
    }
    for (auto it = g_big.begin(); it != g_big.end();) {
        if (it->second.device == device) it = g_big.erase(it);
        else ++it;
    }
    return id;
}

// A kept block of at most a quarter more than asked for, or NULL.
void* take_kept(size_t bytes, int device)
{
    std::lock_guard<std::mutex> lock(g_mem_mutex);
    int best = -1;
    for (int i = 0; i < (int)g_kept.size(); i++)
        if (g_kept[i].device == device && g_kept[i].bytes >= bytes && g_kept[i].bytes <= bytes + bytes / 4 &&
            (best < 0 || g_kept[i].bytes < g_kept[best].bytes))
            best = i;
    if (best < 0) return nullptr;
    const BigBlock b = g_kept[best];
    g_kept.erase(g_kept.begin() + best);
    g_big[b.p] = b;
    return b.p;
}

void drop_kept(int device)
{
    std::vector<BigBlock> drop;
    {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        for (size_t i = 0; i < g_kept.size();) {
            if (g_kept[i].device != device) { i++; continue; }
            drop.push_back(g_kept[i]);
            g_kept.erase(g_kept.begin() + i);
        }
    }
    for (const BigBlock& b : drop) cudaFree(b.p);
}

cudaMemPool_t pool_of(int device)
{
    if (device < 0 || device >= PBB_MEM_DEVICES) return nullptr;
    std::lock_guard<std::mutex> lock(g_mem_mutex);
    if (!g_pool_tried[device]) {
        g_pool_tried[device] = true;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        unsigned long long keep = PBB_POOL_KEEP;
        if (cudaMemPoolCreate(&p, &props) == cudaSuccess &&
            cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
            g_pool[device] = p;
        else
            cudaGetLastError();      // no pools here: plain allocations
    }
    return g_pool[device];
}

}  // namespace

namespace pbbh {

void mem_release(int device)
{
    check_context(device);
    drop_kept(device);
    cudaMemPool_t p = nullptr;
    std::vector<cudaStream_t> streams;
    if (device >= 0 && device < PBB_MEM_DEVICES) {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        p = g_pool[device];
        streams.swap(g_streams[device]);
    }
    // frees still in a stream's order come before the pool can shrink
    for (cudaStream_t st : streams) {
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
    }
    if (p) cudaMemPoolTrimTo(p, 0);
    cudaGetLastError();
}

bool alive(const Lease& l) { return l.st && context_id() == l.context; }

cudaError_t mem_alloc(void** out, size_t bytes, const Lease& l)
{
    *out = nullptr;
    const int device = l.device;
    if (check_context(device) != l.context) return cudaErrorInvalidResourceHandle;
    const bool big = bytes > PBB_BIG_BLOCK;
    cudaMemPool_t p = pool_of(device);
    cudaError_t rc = cudaErrorMemoryAllocation;
    for (int attempt = 0; attempt < 2 && rc != cudaSuccess; attempt++) {
        if (attempt == 1) {
            // what is kept goes back before an allocation fails
            cudaGetLastError();
            mem_release(device);
        }
        if (big) {
            if ((*out = take_kept(bytes, device))) return cudaSuccess;
            rc = cudaMalloc(out, bytes);
        } else {
            rc = p ? cudaMallocFromPoolAsync(out, bytes, p, l.st) : cudaMalloc(out, bytes);
        }
    }
    if (rc == cudaSuccess && big) {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        g_big[*out] = BigBlock{*out, bytes, device};
    }
    return rc;
}

void mem_free(void* p, const Lease& l)
{
    if (!p || !alive(l)) return;
    bool big = false;
    {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        auto it = g_big.find(p);
        if (it != g_big.end()) {
            const BigBlock b = it->second;
            g_big.erase(it);
            big = true;
            size_t kept = b.bytes;
            for (const BigBlock& k : g_kept)
                if (k.device == b.device) kept += k.bytes;
            if (kept <= PBB_BIG_KEEP) {
                g_kept.push_back(b);
                return;
            }
        }
    }
    if (!big) {
        if (cudaFreeAsync(p, l.st) == cudaSuccess) return;
        cudaGetLastError();
    }
    cudaFree(p);
}

cudaError_t stream_take(Lease* l, int device)
{
    l->device = device;
    l->context = check_context(device);
    if (device >= 0 && device < PBB_MEM_DEVICES) {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        if (!g_streams[device].empty()) {
            // its last user's frees may still be on it: they come before the
            // next user's work, as any order of the stream does
            l->st = g_streams[device].back();
            g_streams[device].pop_back();
            return cudaSuccess;
        }
    }
    l->st = nullptr;
    return cudaStreamCreateWithFlags(&l->st, cudaStreamNonBlocking);
}

void stream_give(Lease& l)
{
    const cudaStream_t st = l.st;
    const bool valid = alive(l);
    l.st = nullptr;
    if (!valid) return;
    if (l.device >= 0 && l.device < PBB_MEM_DEVICES) {
        std::lock_guard<std::mutex> lock(g_mem_mutex);
        if (g_streams[l.device].size() < PBB_STREAMS_KEPT) {
            g_streams[l.device].push_back(st);
            return;
        }
    }
    cudaStreamDestroy(st);
}

}  // namespace pbbh
