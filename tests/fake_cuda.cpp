// A CUDA runtime on host memory, for the library's host code without a GPU
// (tests/test_host_faults.py links it with the host files of the library): it
// keeps account of blocks, streams and contexts, fails the calls it is told to
// fail, and counts uses of handles that are not valid.  The kernel launches it
// stands in for only move enough data to tell right from stale inputs.
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "pbb_types.h"
#include "pbb_launch.h"
#include "pbb_heur.h"

namespace {
std::recursive_mutex g_mu;
typedef std::lock_guard<std::recursive_mutex> Lock;

struct Mem {
    size_t bytes;
    unsigned long long context;
    bool pooled;
};
struct FakeStream {
    unsigned long long context;
    bool busy;
};
unsigned long long g_ctx = 1;
std::map<void*, Mem> g_mem;
std::set<FakeStream*> g_streams;
std::vector<void*> g_spare;                // addresses of the contexts before, handed out again first
std::map<std::string, int> g_fail, g_calls;
size_t g_capacity = ~(size_t)0, g_used = 0, g_reserved = 0, g_threshold = 0;
int g_invalid = 0;                         // uses of handles that are not valid
int g_variant = -1, g_eager = -1;
int g_windows = 1;                         // windows a search takes
int g_per_sm[8] = {2, 2, 2, 2, 2, 2, 2, 2};   // resident CTAs an SM, by explorer variant
int g_not_resident = 0;                    // explorer launches of more CTAs than are resident
cudaError_t g_last = cudaSuccess;

cudaError_t done(const char* name, cudaError_t rc = cudaSuccess)
{
    g_calls[name]++;
    auto it = g_fail.find(name);
    if (it != g_fail.end() && --it->second == 0) {
        g_fail.erase(it);
        rc = cudaErrorInvalidValue;
    }
    if (rc != cudaSuccess) g_last = rc;
    return rc;
}

bool live(cudaStream_t st)
{
    FakeStream* s = reinterpret_cast<FakeStream*>(st);
    const bool ok = g_streams.count(s) && s->context == g_ctx;
    if (!ok) g_invalid++;
    return ok;
}

cudaError_t take(void** p, size_t bytes, bool pooled)
{
    const size_t from_pool = pooled ? (g_reserved < bytes ? g_reserved : bytes) : 0;
    if (g_used + g_reserved - from_pool + bytes > g_capacity) return cudaErrorMemoryAllocation;
    g_reserved -= from_pool;
    g_used += bytes;
    *p = nullptr;
    for (size_t i = 0; i < g_spare.size() && !*p; i++)
        if (g_mem[g_spare[i]].bytes >= bytes) {
            *p = g_spare[i];
            g_spare.erase(g_spare.begin() + i);
        }
    if (!*p) *p = calloc(1, bytes ? bytes : 1);
    g_mem[*p] = Mem{bytes, g_ctx, pooled};
    return cudaSuccess;
}

cudaError_t give(void* p, bool pooled)
{
    auto it = g_mem.find(p);
    if (it == g_mem.end() || it->second.context != g_ctx) {
        g_invalid++;
        return cudaErrorInvalidValue;
    }
    g_used -= it->second.bytes;
    if (pooled && it->second.pooled) {
        g_reserved += it->second.bytes;
        if (g_reserved > g_threshold) g_reserved = g_threshold;
    }
    g_mem.erase(it);
    free(p);
    return cudaSuccess;
}

cudaError_t copy(const char* name, void* to, const void* from, size_t bytes)
{
    const cudaError_t rc = done(name);
    if (rc == cudaSuccess) memcpy(to, from, bytes);
    return rc;
}

int fake_get_id(void*, unsigned long long* id) { *id = g_ctx; return 0; }
int fake_get_current(void** c) { *c = nullptr; return 0; }
int fake_set_current(void*) { return 0; }
}  // namespace

extern "C" {
// --- control --------------------------------------------------------------
// the nth call of `name` from here on fails
void fake_fail(const char* name, int nth) { Lock l(g_mu); g_fail[name] = nth; }
void fake_capacity(size_t bytes) { Lock l(g_mu); g_capacity = bytes; }
// the device is reset: every handle dies, its addresses are handed out again
void fake_reset()
{
    Lock l(g_mu);
    for (auto& m : g_mem)
        if (m.second.context == g_ctx) g_spare.push_back(m.first);
    g_used = g_reserved = 0;
    g_ctx++;
}
int fake_invalid() { Lock l(g_mu); return g_invalid; }
void fake_per_sm(int variant, int ctas) { Lock l(g_mu); g_per_sm[variant] = ctas; }
int fake_not_resident() { Lock l(g_mu); return g_not_resident; }
int fake_eager() { Lock l(g_mu); return g_eager; }
void fake_windows(int n) { Lock l(g_mu); g_windows = n; }
int fake_variant() { Lock l(g_mu); return g_variant; }
size_t fake_used() { Lock l(g_mu); return g_used + g_reserved; }
int fake_calls(const char* name) { Lock l(g_mu); return g_calls[name]; }
int fake_streams()
{
    Lock l(g_mu);
    int n = 0;
    for (FakeStream* s : g_streams) n += s->context == g_ctx;
    return n;
}

// --- runtime ----------------------------------------------------------------
cudaError_t cudaGetLastError(void) { Lock l(g_mu); const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 148;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q)
{
    const std::string n = name;
    *f = n == "cuCtxGetId" ? (void*)fake_get_id : n == "cuCtxGetCurrent" ? (void*)fake_get_current
                                                                        : (void*)fake_set_current;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n)
{
    Lock l(g_mu);
    const cudaError_t rc = done("cudaMalloc");
    return rc ? rc : done("", take(p, n, false));
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    const cudaError_t rc = done("cudaMallocFromPoolAsync");
    return rc ? rc : done("", take(p, n, true));
}
cudaError_t cudaFree(void* p)
{
    Lock l(g_mu);
    return p ? done("cudaFree", give(p, false)) : cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    reinterpret_cast<FakeStream*>(st)->busy = true;
    return done("cudaFreeAsync", give(p, true));
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*)
{
    *p = reinterpret_cast<cudaMemPool_t>(0x10);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void* v)
{
    Lock l(g_mu);
    g_threshold = (size_t)*reinterpret_cast<unsigned long long*>(v);
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t n)
{
    Lock l(g_mu);
    if (g_reserved > n) g_reserved = n;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned)
{
    Lock l(g_mu);
    const cudaError_t rc = done("cudaStreamCreateWithFlags");
    if (rc) return rc;
    FakeStream* s = new FakeStream{g_ctx, false};
    g_streams.insert(s);
    *st = reinterpret_cast<cudaStream_t>(s);
    return rc;
}
cudaError_t cudaStreamDestroy(cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    g_streams.erase(reinterpret_cast<FakeStream*>(st));
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    return done("cudaStreamQuery", reinterpret_cast<FakeStream*>(st)->busy ? cudaErrorNotReady : cudaSuccess);
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    reinterpret_cast<FakeStream*>(st)->busy = false;
    return done("cudaStreamSynchronize");
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, enum cudaMemcpyKind)
{
    Lock l(g_mu);
    return copy("cudaMemcpy", to, from, n);
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, enum cudaMemcpyKind, cudaStream_t st)
{
    Lock l(g_mu);
    return live(st) ? copy("cudaMemcpyAsync", to, from, n) : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st)
{
    Lock l(g_mu);
    if (!live(st)) return cudaErrorInvalidResourceHandle;
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(0x20); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
// a graph is the launches and copies of its capture: none here, the calls
// made in it have had their effect
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = reinterpret_cast<cudaGraph_t>(0x30); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long)
{
    Lock l(g_mu);
    *e = reinterpret_cast<cudaGraphExec_t>(0x40);
    return done("cudaGraphInstantiate");
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}  // extern "C"

// --- launches ---------------------------------------------------------------
namespace pbbl {
int smem_bytes(int n, int m, int Ppad, int warps, int fmask) { return pbb_smem_plan(n, m, Ppad, warps, fmask).total; }
cudaError_t launch_reset(const DevGroup*, int, const int*, cudaStream_t) { return cudaSuccess; }
int explore_ctas_per_sm(int, int, int, int variant) { return g_per_sm[variant]; }
cudaError_t launch_root(int, const DevGroup* g, int count, const int*, const int*, int, int, cudaStream_t, int, const int*)
{
    for (int i = 0; i < count; i++) g[i].ctl->active = 1;
    return cudaSuccess;
}
cudaError_t launch_lower_ub(const DevGroup*, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_explore(int, const DevGroup* g, const int* count, int ctas, int, int, unsigned long long, int, int,
                           cudaStream_t, int variant, int eager, int*, int)
{
    Lock l(g_mu);
    g_variant = variant;
    g_eager = eager;
    g_not_resident += ctas > 148 * g_per_sm[variant];
    if (--g_windows <= 0)
        for (int i = 0; i < *count; i++) g[i].ctl->active = 0;
    return cudaSuccess;
}
cudaError_t launch_neh(const NehTask*, int, cudaStream_t) { return cudaSuccess; }
BoundShape bound_shape(int, int, int, int, int, int)
{
    BoundShape b;
    b.all = true;
    b.warps = 1;
    return b;
}
// every output depends on the tables, the nodes and both limits
static cudaError_t bounds(const DevInstance& I, int count, const int* s, const int* l1, const int* l2, int* wb, int* we,
                          int* sb, int* se, int* nw, int* ns, const BoundExtra& X)
{
    int sum = 0;
    for (int i = 0; i < I.n * I.m; i++) sum = 31 * sum + I.p[i];
    for (int i = 0; i < count; i++) {
        int x = sum + 7 * l1[i] + 13 * l2[i];
        for (int t = 0; t < I.n; t++) x = 17 * x + s[i * I.n + t];
        for (int t = 0; t < I.n; t++) {
            wb[i * I.n + t] = x + t;
            we[i * I.n + t] = x + 2 * t;
            sb[i * I.n + t] = x + 3 * t;
            se[i * I.n + t] = x + 4 * t;
            if (X.prio_begin) X.prio_begin[i * I.n + t] = x + 5 * t;
            if (X.prio_end) X.prio_end[i * I.n + t] = x + 6 * t;
        }
        nw[i] = x;
        ns[i] = x + 1;
        if (X.strong_idle) X.strong_idle[i] = x + 2;
    }
    return cudaSuccess;
}
cudaError_t launch_bound_all(int, const DevInstance& I, int count, const int* s, const int* l1, const int* l2, int* wb,
                             int* we, int* sb, int* se, int* nw, int* ns, unsigned int*, const BoundShape&, cudaStream_t,
                             BoundExtra X)
{
    return bounds(I, count, s, l1, l2, wb, we, sb, se, nw, ns, X);
}
cudaError_t launch_bound(int, const DevInstance& I, int count, const int* s, const int* l1, const int* l2, int* wb, int* we,
                         int* sb, int* se, int* nw, int* ns, unsigned int*, int, int, int, cudaStream_t, int, BoundExtra X)
{
    return bounds(I, count, s, l1, l2, wb, we, sb, se, nw, ns, X);
}
}  // namespace pbbl
