// Host side of the engine: instance tables, device memory, launches, and the
// C ABI declared in include/pbbperm.h.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <string>
#include <thread>
#include <vector>

#include "pbb_types.h"
#include "pbb_devguard.h"
#include "pbb_launch.h"
#include "pbb_tables.h"
#include "pbb_heur.h"
#include "pbb_mem.h"
#include "../../include/pbbperm.h"
#include "../../include/pbbperm_diag.h"

using pbbt::HostTables;
using pbbt::build_tables;

namespace {

thread_local std::string g_err;

int fail(int code, const std::string& msg)
{
    g_err = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* where)
{
    g_err = std::string(where) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? PBB_E_NOMEM : PBB_E_CUDA;
}

#define CK(call)                                        \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

// An instance's tables as one block, laid out on the host and uploaded by one
// copy.
struct InstanceBlock {
    size_t je, posj, p, pm, mt;       // offsets
    explicit InstanceBlock(const HostTables& H, pbbh::Carver& C)
    {
        je = C.take(sizeof(unsigned long long) * H.je.size());
        posj = C.take(H.posj.size());
        p = C.take(sizeof(int) * H.n * H.m);
        pm = C.take(2 * H.Ppad);
        mt = C.take(sizeof(int) * 2 * H.m);
    }
    void fill(const HostTables& H, unsigned char* host) const
    {
        memcpy(host + je, H.je.data(), sizeof(unsigned long long) * H.je.size());
        memcpy(host + posj, H.posj.data(), H.posj.size());
        memcpy(host + p, H.p.data(), sizeof(int) * H.n * H.m);
        memcpy(host + pm, H.pm0.data(), H.Ppad);
        memcpy(host + pm + H.Ppad, H.pm1.data(), H.Ppad);
        memcpy(host + mt, H.min_arr.data(), sizeof(int) * H.m);
        memcpy(host + mt + sizeof(int) * H.m, H.min_dep.data(), sizeof(int) * H.m);
    }
    DevInstance view(const HostTables& H, unsigned char* dev) const
    {
        DevInstance v{};
        v.n = H.n; v.m = H.m; v.P = H.P; v.Ppad = H.Ppad;
        v.je = reinterpret_cast<const unsigned long long*>(dev + je);
        v.posj = dev + posj;
        v.p = reinterpret_cast<const int*>(dev + p);
        v.pm0 = dev + pm; v.pm1 = dev + pm + H.Ppad;
        v.min_arr = reinterpret_cast<const int*>(dev + mt);
        v.min_dep = v.min_arr + H.m;
        return v;
    }
};

int max_smem_optin(int dev)
{
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

// The most warps per CTA (up to `requested`) whose tables and scratch fit;
// `explorer`: add the per-warp free-position masks when they fit too (the
// explorer runs one CTA per SM, so they never cost a warp).
int pick_warps(const HostTables& H, int requested, int dev, int& smem, bool explorer = false)
{
    const int cap = max_smem_optin(dev);
    int w = requested > 0 ? std::min(requested, PBB_WARPS_MAX) : PBB_WARPS_MAX;
    for (; w >= 1; w--) {
        smem = pbbl::smem_bytes(H.n, H.m, H.Ppad, w);
        if (smem <= cap) {
            const int with_masks = pbbl::smem_bytes(H.n, H.m, H.Ppad, w, 1);
            if (explorer && with_masks <= cap) smem = with_masks;
            return w;
        }
    }
    return 0;
}

}  // namespace

namespace pbbh {
// error message for entry points compiled in other files of the library
void set_error(const char* msg) { g_err = msg; }
}  // namespace pbbh

struct pbb_engine;
namespace pbbh {
// engine facts for the checkpoint code (pbb_ckpt.cu)
int engine_jobs(const pbb_engine* e);
int engine_explorers(const pbb_engine* e);
const std::vector<int32_t>& engine_root(const pbb_engine* e);
void engine_set_start_perm(pbb_engine* e, const int32_t* perm);
}  // namespace pbbh

// ---------------------------------------------------------------------------
// engine
// ---------------------------------------------------------------------------
struct pbb_engine {
    pbb_config cfg{};
    HostTables H;
    int dev = 0;
    pbbh::Lease lease;
    cudaStream_t st = nullptr;        // the lease's
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    int nw = 2, warps = 0, ctas = 0, smem = 0, root_smem = 0;
    // the launch of the explorer variants 3 to 7, pair_warps 0: not used
    int pair_variant = 0, pair_warps = 0, pair_smem = 0, pair_stride = 0;
    int* pair_stack = nullptr;
    unsigned char* block = nullptr;   // everything below but the pair bounds and samples
    int npad = 32;                    // row stride
    signed char* bestperm = nullptr;
    int *state = nullptr, *ub_d = nullptr, *root_d = nullptr;
    int* ival_d = nullptr;   // [2][64] interval start / end vectors
    GroupCtl* ctl = nullptr;
    DevGroup* group_d = nullptr;
    int* ngroups_d = nullptr;     // device copy of the group count (1)
    DevGroup group{};
    double dev_seconds = 0.0;
    bool started = false, done = false;
    int32_t ub = INT32_MAX;
    double slice_s = 2.0;
    int select_budget = 4096;
    int max_rounds = INT_MAX;      // explorer loop rounds per launch
    int* neh_d = nullptr;          // device NEH result: perm[64], cost
    NehTask* neh_task_d = nullptr; // the engine's instance as a heuristic task
    bool from_neh = false;         // the current search started from PBB_UB_NEH
    std::vector<int32_t> root;     // root permutation of the current search
    std::vector<int32_t> start_perm;   // schedule of the starting bound (e.g. a checkpoint's incumbent)
    SampleBuf* sample_d = nullptr; // node sampling (diagnostic), NULL when off
    int* sample_rec = nullptr;
    int sample_stride = 0;
    bool sample_decisions = false; // by the build with kept pair bounds
    double wait_limit_s = -1.0;    // host wait per window: < 0 window + 60 s, 0 unbounded
    bool pending = false;          // a window whose wait ran out is still on the stream
    bool exporting = true;         // the search has just started, or its intervals were exported since its last window
};

namespace pbbh {
int engine_jobs(const pbb_engine* e) { return e->H.n; }
int engine_explorers(const pbb_engine* e) { return e->cfg.nb_ivms; }
const std::vector<int32_t>& engine_root(const pbb_engine* e) { return e->root; }
void engine_set_start_perm(pbb_engine* e, const int32_t* perm) { e->start_perm.assign(perm, perm + e->H.n); }
}  // namespace pbbh

namespace {

// Wait for `ev` with a host-side deadline: PBB_E_TIMEOUT when it has not
// completed after limit_s seconds (limit_s <= 0: wait without limit).  Polls
// with a short sleep so that the waiting thread does not spin a core.
int wait_event(cudaEvent_t ev, double limit_s)
{
    if (limit_s <= 0) {
        CK(cudaEventSynchronize(ev));
        return PBB_OK;
    }
    const auto t0 = std::chrono::steady_clock::now();
    while (true) {
        const cudaError_t q = cudaEventQuery(ev);
        if (q == cudaSuccess) return PBB_OK;
        if (q != cudaErrorNotReady) return cuda_fail(q, "exploration window");
        const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (el > limit_s) return PBB_E_TIMEOUT;
        // small searches end within a fraction of a millisecond; later on the
        // pause is a sixteenth of the time waited
        if (el < 5e-4) std::this_thread::yield();
        else std::this_thread::sleep_for(std::chrono::microseconds((int)std::min(el * 1e6 / 16, 500.0)));
    }
}

// Account a window whose host wait ran out: it ends by its own device-time
// budget, so this blocks for at most the rest of that budget.
int settle(pbb_engine* e)
{
    if (!e->pending) return PBB_OK;
    CK(cudaEventSynchronize(e->ev1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e->ev0, e->ev1));
    e->dev_seconds += ms * 1e-3;
    int active = 0;
    CK(cudaMemcpy(&active, &e->ctl->active, sizeof(int), cudaMemcpyDeviceToHost));
    e->done = (active == 0);
    e->pending = false;
    return PBB_OK;
}

}  // namespace

extern "C" {

void pbb_config_default(pbb_config* c)
{
    if (!c) return;
    memset(c, 0, sizeof(*c));
    c->bounding_mode = 2;
    c->branching_mode = 3;
    c->find_all = 0;
    c->johnson_mode = 0;
    c->early_stop_johnson = 0;
    c->sorted_dfs = 0;
    c->sorting_criterion = 1;
    c->nb_ivms = 16384;
    c->device = 0;
}

const char* pbb_last_error(void) { return g_err.c_str(); }

int pbb_release_memory(int32_t device)
{
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(device));
    pbbh::mem_release(device);
    return PBB_OK;
}

}  // extern "C"

namespace pbbh {
// Search settings every entry point accepts (engine and pool).
// earlyStopJohnson: a child's Johnson scan stops once its running maximum
// exceeds the incumbent (bound_fsp_strong.cpp:154-158); that child is pruned
// either way, so node counts do not change -- except with the Johnson bound
// choosing the side by MaxSum (boundingMode 1, adaptiveBranchingMode 1),
// where the pruned children's partial values enter the choice and, in the
// reference, depend on each thread's machine-pair success history
// (:112-122): that combination is rejected.
int check_search(const pbb_config* c)
{
    if (c->bounding_mode < 0 || c->bounding_mode > 2) return fail(PBB_E_INVAL, "boundingMode must be 0, 1 or 2");
    const int b = c->branching_mode;
    if (!(b == -3 || b == -2 || b == -1 || b == 1 || b == 2 || b == 3))
        return fail(PBB_E_INVAL, "adaptiveBranchingMode must be one of -3,-2,-1,1,2,3");
    if (c->early_stop_johnson && c->bounding_mode == 1 && b == 1)
        return fail(PBB_E_UNSUPPORTED, "earlyStopJohnson=true with boundingMode=1 and MaxSum branching is not "
                                       "supported (the side choice would depend on a thread's pair-order history)");
    if (c->sorted_dfs < 0 || c->sorted_dfs > 4) return fail(PBB_E_INVAL, "sortedDFS must be in 0..4");
    if (c->sorted_dfs >= 2) {
        // the sibling priorities of chooseChildrenSet (ivm_bound.cpp:506-544)
        const int k = c->sorting_criterion;
        if (k == 4)
            return fail(PBB_E_UNSUPPORTED, "sortingCriterion=4 is not supported: the reference's completeSchedule "
                                           "writes past the node's free jobs, so its priorities are not defined");
        if (k < 1 || k > 4) return fail(PBB_E_INVAL, "sortingCriterion must be 1, 2 or 3 with sortedDFS >= 2");
        if (k == 3 && c->bounding_mode == 1)
            return fail(PBB_E_UNSUPPORTED, "sortingCriterion=3 with boundingMode=1 is not supported: the reference "
                                           "reads an unset Johnson idle time for children with one free job");
        if (k == 2 && c->bounding_mode == 1 && c->early_stop_johnson)
            return fail(PBB_E_UNSUPPORTED, "sortingCriterion=2 with boundingMode=1 and earlyStopJohnson=true is not "
                                           "supported: the priority would read a pruned side's partial bound");
    }
    return PBB_OK;
}
}  // namespace pbbh

extern "C" {

static int check_config(const pbb_config* c)
{
    const int rc = pbbh::check_search(c);
    if (rc) return rc;
    if (c->nb_ivms < 1 || c->nb_ivms > (1 << 22)) return fail(PBB_E_INVAL, "nbIVMs must be in [1, 4194304]");
    return PBB_OK;
}

int pbb_engine_destroy(pbb_engine* e)
{
    if (!e) return PBB_OK;
    pbbh::DeviceGuard keep_callers_device;
    cudaSetDevice(e->dev);
    if (pbbh::alive(e->lease)) {
        cudaStreamSynchronize(e->st);
        pbbh::mem_free(e->block, e->lease);
        pbbh::mem_free(e->pair_stack, e->lease);
        pbbh::mem_free(e->sample_d, e->lease);
        pbbh::mem_free(e->sample_rec, e->lease);
        if (e->ev0) cudaEventDestroy(e->ev0);
        if (e->ev1) cudaEventDestroy(e->ev1);
        pbbh::stream_give(e->lease);
    }
    delete e;
    return PBB_OK;
}

static int engine_create(const pbb_instance* inst, const pbb_config* cfg, pbb_engine* e)
{
    e->cfg = *cfg;
    int rc = check_config(cfg);
    if (rc) return rc;
    rc = build_tables(inst, cfg->johnson_mode, e->H);
    if (rc) return rc;
    e->dev = cfg->device;
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    CK(pbbh::stream_take(&e->lease, e->dev));
    e->st = e->lease.st;
    CK(cudaEventCreate(&e->ev0));
    CK(cudaEventCreate(&e->ev1));
    const HostTables& H = e->H;
    e->nw = H.n <= 32 ? 1 : 2;
    e->warps = pick_warps(H, cfg->warps_per_cta, e->dev, e->smem, true);
    if (e->warps < 1) return fail(PBB_E_INVAL, "instance tables do not fit in shared memory");
    e->root_smem = pbbl::smem_bytes(H.n, H.m, H.Ppad, 1);
    int sms = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->dev));
    e->ctas = cfg->ctas > 0 ? cfg->ctas : sms;
    e->pair_variant = pbbl::pairs_variant(cfg->bounding_mode, cfg->branching_mode, cfg->find_all, cfg->sorted_dfs);
    if (e->pair_variant) {
        // earlyStopJohnson changes the values of pruned children only, which
        // these builds do not compute: they serve both settings
        const int cap = max_smem_optin(e->dev);
        // (instances whose tables hold the general build below its full CTA
        // keep that count in every build: the work statistics report one)
        const bool wide = cfg->warps_per_cta <= 0 && e->warps == PBB_WARPS_MAX && H.n * H.m > PBB_WIDE_FROM;
        if (wide) e->pair_variant += 2;
        int w = wide ? PBB_WIDE_WARPS : e->warps;
        while (w > 1 && pbbl::smem_bytes(H.n, H.m, H.Ppad, w, PBB_SCRATCH_PAIRS) > cap) w--;
        e->pair_smem = pbbl::smem_bytes(H.n, H.m, H.Ppad, w, PBB_SCRATCH_PAIRS);
        e->pair_stride = H.n * H.Ppad;
        if (e->pair_smem <= cap) e->pair_warps = w;
    }
    // mode 1: the general build's shared atomics against values by position, at
    // the same warps (24 gain 7 % on 20x20 and lose 2 to 4 % on 18x20 to 30x10)
    if (cfg->bounding_mode == 1 && e->nw == 1) {
        e->pair_smem = pbbl::smem_bytes(H.n, H.m, H.Ppad, e->warps, PBB_SCRATCH_ALL);
        if (e->pair_smem <= max_smem_optin(e->dev)) {
            e->pair_variant = 7;
            e->pair_warps = e->warps;
        }
    }
    // one block: what the host fills first (one upload), then the explorers
    const size_t B = (size_t)cfg->nb_ivms;
    const size_t npad = e->npad = 32 * e->nw, levels = H.n;
    pbbh::Carver C;
    const InstanceBlock tables(H, C);
    const size_t o_group = C.take(sizeof(DevGroup)), o_one = C.take(sizeof(int)), o_task = C.take(sizeof(NehTask));
    const size_t filled = C.bytes;
    const size_t o_ub = C.take(sizeof(int)), o_root = C.take(sizeof(int) * PBB_MAX_N);
    const size_t o_ival = C.take(sizeof(int) * 2 * PBB_MAX_N), o_neh = C.take(sizeof(int) * (PBB_MAX_N + 1));
    const size_t o_ctl = C.take(sizeof(GroupCtl));
    const size_t o_line = C.take(sizeof(int) * B), o_state = C.take(sizeof(int) * B);
    const size_t o_cost = C.take(sizeof(int) * B), o_askid = C.take(sizeof(int) * B);
    const size_t o_ask = C.take(sizeof(unsigned) * ((B + 31) / 32));
    const size_t o_vec = C.take(4 * B * npad), o_perm = C.take(B * npad);
    const size_t o_mat = C.take(B * levels * npad), o_path = C.take(B * levels * PBB_PATH_INTS * sizeof(int));
    // the pair bounds stand before the explorers in the store (20x10: 0.890 ms of
    // device time, 0.916 behind them), but go back if those do not fit as well:
    // the general build needs none
    if (e->pair_warps > 0 && PBB_VAR_PAIRS(e->pair_variant) &&
        pbbh::mem_alloc((void**)&e->pair_stack, sizeof(int) * (size_t)e->ctas * e->pair_warps * e->pair_stride,
                        e->lease) != cudaSuccess) {
        cudaGetLastError();
        e->pair_warps = 0;
    }
    cudaError_t room = pbbh::mem_alloc((void**)&e->block, C.bytes, e->lease);
    if (room == cudaErrorMemoryAllocation && e->pair_stack) {
        cudaGetLastError();
        pbbh::mem_free(e->pair_stack, e->lease);
        CK(cudaStreamSynchronize(e->st));
        e->pair_stack = nullptr;
        e->pair_warps = 0;
        room = pbbh::mem_alloc((void**)&e->block, C.bytes, e->lease);
    }
    CK(room);
    unsigned char* d = e->block;
    e->ub_d = reinterpret_cast<int*>(d + o_ub);
    e->root_d = reinterpret_cast<int*>(d + o_root);
    e->ival_d = reinterpret_cast<int*>(d + o_ival);
    e->neh_d = reinterpret_cast<int*>(d + o_neh);
    e->neh_task_d = reinterpret_cast<NehTask*>(d + o_task);
    e->ctl = reinterpret_cast<GroupCtl*>(d + o_ctl);
    e->group_d = reinterpret_cast<DevGroup*>(d + o_group);
    e->ngroups_d = reinterpret_cast<int*>(d + o_one);
    e->state = reinterpret_cast<int*>(d + o_state);
    e->bestperm = reinterpret_cast<signed char*>(d + o_perm);
    DevGroup& g = e->group;
    g.inst = tables.view(H, d);
    g.search.bound_mode = cfg->bounding_mode;
    g.search.branch_mode = cfg->branching_mode;
    g.search.find_all = cfg->find_all ? 1 : 0;
    g.search.sort_nodes = cfg->sorted_dfs;
    g.search.sort_crit = cfg->sorting_criterion;
    g.search.core_warps = cfg->core_warps > 0 ? cfg->core_warps : PBB_CORE_WARPS;
    g.search.split_depth = cfg->split_depth > 0 ? cfg->split_depth : PBB_SPLIT_DEPTH;
    g.search.split_narrow = cfg->split_depth > 0 ? cfg->split_depth : PBB_SPLIT_NARROW;
    g.search.share_after = cfg->share_after > 0 ? cfg->share_after : (cfg->share_after < 0 ? 0 : PBB_SHARE_AFTER);
    g.search.early_stop = cfg->early_stop_johnson ? 1 : 0;
    g.ivm.count = cfg->nb_ivms;
    g.ivm.npad = e->npad;
    g.ivm.levels = H.n;
    g.ivm.mat = reinterpret_cast<signed char*>(d + o_mat);
    g.ivm.pos = reinterpret_cast<signed char*>(d + o_vec);
    g.ivm.end = g.ivm.pos + B * npad;
    g.ivm.dir = g.ivm.end + B * npad;
    g.ivm.pj = g.ivm.dir + B * npad;
    g.ivm.line = reinterpret_cast<int*>(d + o_line);
    g.ivm.state = e->state;
    g.ivm.bestcost = reinterpret_cast<int*>(d + o_cost);
    g.ivm.bestperm = e->bestperm;
    g.ivm.ask = reinterpret_cast<unsigned*>(d + o_ask);
    g.ivm.askid = reinterpret_cast<int*>(d + o_askid);
    g.ivm.path = reinterpret_cast<int*>(d + o_path);
    g.ctl = e->ctl;
    g.first_cta = 0;
    g.ctas = e->ctas;
    g.sample = nullptr;
    NehTask t;
    t.p = g.inst.p;
    t.n = H.n;
    t.m = H.m;
    t.perm = e->neh_d;
    t.cost = e->neh_d + PBB_MAX_N;
    t.ub = e->ub_d;
    const int one = 1;
    std::vector<unsigned char> host(filled);
    tables.fill(H, host.data());
    memcpy(host.data() + o_group, &g, sizeof(g));
    memcpy(host.data() + o_one, &one, sizeof(one));
    memcpy(host.data() + o_task, &t, sizeof(t));
    CK(cudaMemcpyAsync(d, host.data(), filled, cudaMemcpyHostToDevice, e->st));
    CK(cudaStreamSynchronize(e->st));
    return PBB_OK;
}

int pbb_engine_create(const pbb_instance* inst, const pbb_config* cfg, pbb_engine** out)
{
    if (!out) return fail(PBB_E_INVAL, "out is NULL");
    *out = nullptr;
    pbb_config def;
    if (!cfg) { pbb_config_default(&def); cfg = &def; }
    pbb_engine* e = new pbb_engine();
    int rc = engine_create(inst, cfg, e);
    if (rc) {
        std::string keep = g_err;
        pbb_engine_destroy(e);
        g_err = keep;
        return rc;
    }
    *out = e;
    return PBB_OK;
}

static int start_impl(pbb_engine* e, int32_t ub, const int32_t* root_perm, const int32_t* pos, const int32_t* end)
{
    if (!e) return fail(PBB_E_INVAL, "engine is NULL");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    const int n = e->H.n;
    std::vector<int> root(PBB_MAX_N, 0);
    std::vector<int> seen(n, 0);
    for (int i = 0; i < n; i++) {
        const int j = root_perm ? root_perm[i] : i;
        if (j < 0 || j >= n || seen[j]) return fail(PBB_E_INVAL, "root_perm is not a permutation of 0..n-1");
        seen[j] = 1;
        root[i] = j;
    }
    // factoradic interval: digit i in [0, n-i) (sequentialbb.cpp:207-222 checks)
    std::vector<int> iv(2 * PBB_MAX_N, 0);
    for (int i = 0; i < n; i++) {
        const int p = pos ? pos[i] : 0;
        const int q = end ? end[i] : n - 1 - i;
        if (p < 0 || p >= n - i || q < 0 || q >= n - i) return fail(PBB_E_INVAL, "interval digit out of range");
        iv[i] = p;
        iv[PBB_MAX_N + i] = q;
    }
    if (ub < 0 && ub != PBB_UB_NEH) return fail(PBB_E_INVAL, "ub must be >= 0 (or PBB_UB_NEH)");
    e->ub = ub;
    e->from_neh = ub == PBB_UB_NEH;
    e->root.assign(root.begin(), root.begin() + n);
    e->start_perm.clear();
    CK(cudaMemcpyAsync(e->ub_d, &ub, sizeof(int), cudaMemcpyHostToDevice, e->st));
    // the device NEH writes its makespan where the reset kernel reads the bound
    if (e->from_neh) CK(pbbl::launch_neh(e->neh_task_d, 1, e->st));
    CK(cudaMemcpyAsync(e->root_d, root.data(), sizeof(int) * PBB_MAX_N, cudaMemcpyHostToDevice, e->st));
    CK(cudaMemcpyAsync(e->ival_d, iv.data(), sizeof(int) * 2 * PBB_MAX_N, cudaMemcpyHostToDevice, e->st));
    CK(pbbl::launch_reset(e->group_d, 1, e->ub_d, e->st));
    CK(pbbl::launch_root(e->nw, e->group_d, 1, e->root_d, e->ival_d, PBB_MAX_N, e->root_smem, e->st));
    CK(cudaStreamSynchronize(e->st));
    if (e->from_neh) CK(cudaMemcpy(&e->ub, e->ub_d, sizeof(int), cudaMemcpyDeviceToHost));
    e->pending = false;
    GroupCtl c;
    CK(cudaMemcpy(&c, e->ctl, sizeof(c), cudaMemcpyDeviceToHost));
    e->started = true;
    e->exporting = true;
    e->done = (c.active == 0);
    e->dev_seconds = 0.0;
    return PBB_OK;
}

int pbb_start(pbb_engine* e, int32_t ub, const int32_t* root_perm) { return start_impl(e, ub, root_perm, nullptr, nullptr); }

int pbb_start_interval(pbb_engine* e, int32_t ub, const int32_t* root_perm, const int32_t* pos, const int32_t* end)
{
    if (!pos || !end) return fail(PBB_E_INVAL, "pos/end are NULL");
    return start_impl(e, ub, root_perm, pos, end);
}

int pbb_init_from_fac(pbb_engine* e, int32_t ub, const int32_t* root_perm, int32_t nb_intervals, const int32_t* ids,
                      const int32_t* pos, const int32_t* end)
{
    if (!e) return fail(PBB_E_INVAL, "engine is NULL");
    if (!pos || !end) return fail(PBB_E_INVAL, "pos/end are NULL");
    const int B = e->cfg.nb_ivms;
    if (nb_intervals < 1 || nb_intervals > B) return fail(PBB_E_INVAL, "nb_intervals must be in [1, nb_ivms]");
    if (ub < 0 && ub != PBB_UB_NEH) return fail(PBB_E_INVAL, "ub must be >= 0 (or PBB_UB_NEH)");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    const int n = e->H.n;
    std::vector<int> root(PBB_MAX_N, 0);
    std::vector<int> seen(n, 0);
    for (int i = 0; i < n; i++) {
        const int j = root_perm ? root_perm[i] : i;
        if (j < 0 || j >= n || seen[j]) return fail(PBB_E_INVAL, "root_perm is not a permutation of 0..n-1");
        seen[j] = 1;
        root[i] = j;
    }
    std::vector<int> iv((size_t)2 * nb_intervals * PBB_MAX_N, 0);
    std::vector<int> id(nb_intervals);
    std::vector<char> taken(B, 0);
    for (int k = 0; k < nb_intervals; k++) {
        const int x = ids ? ids[k] : k;
        if (x < 0 || x >= B || taken[x]) return fail(PBB_E_INVAL, "ids must be distinct explorers < nb_ivms");
        taken[x] = 1;
        id[k] = x;
        for (int i = 0; i < n; i++) {
            const int p = pos[(size_t)k * n + i], q = end[(size_t)k * n + i];
            if (p < 0 || p >= n - i || q < 0 || q >= n - i) return fail(PBB_E_INVAL, "interval digit out of range");
            iv[(size_t)(2 * k) * PBB_MAX_N + i] = p;
            iv[(size_t)(2 * k + 1) * PBB_MAX_N + i] = q;
        }
    }
    const size_t iv_bytes = sizeof(int) * iv.size(), id_bytes = sizeof(int) * nb_intervals;
    int* ival_d = nullptr;
    CK(pbbh::mem_alloc((void**)&ival_d, iv_bytes + id_bytes, e->lease));
    int* ids_d = ival_d + iv.size();
    cudaError_t err = cudaMemcpyAsync(ival_d, iv.data(), iv_bytes, cudaMemcpyHostToDevice, e->st);
    if (!err) err = cudaMemcpyAsync(ids_d, id.data(), sizeof(int) * nb_intervals, cudaMemcpyHostToDevice, e->st);
    if (!err) err = cudaMemcpyAsync(e->ub_d, &ub, sizeof(int), cudaMemcpyHostToDevice, e->st);
    if (!err && ub == PBB_UB_NEH) err = pbbl::launch_neh(e->neh_task_d, 1, e->st);
    if (!err) err = cudaMemcpyAsync(e->root_d, root.data(), sizeof(int) * PBB_MAX_N, cudaMemcpyHostToDevice, e->st);
    if (!err) err = pbbl::launch_reset(e->group_d, 1, e->ub_d, e->st);
    if (!err)
        err = pbbl::launch_root(e->nw, e->group_d, 1, e->root_d, ival_d, PBB_MAX_N, e->root_smem, e->st,
                                nb_intervals, ids_d);
    if (!err) err = cudaStreamSynchronize(e->st);
    if (!err) e->pending = false;
    pbbh::mem_free(ival_d, e->lease);
    if (err) return fail(PBB_E_CUDA, std::string("init_from_fac: ") + cudaGetErrorString(err));
    GroupCtl c;
    CK(cudaMemcpy(&c, e->ctl, sizeof(c), cudaMemcpyDeviceToHost));
    e->ub = ub;
    e->from_neh = ub == PBB_UB_NEH;
    if (e->from_neh) CK(cudaMemcpy(&e->ub, e->ub_d, sizeof(int), cudaMemcpyDeviceToHost));
    e->root.assign(root.begin(), root.begin() + n);
    e->start_perm.clear();
    e->started = true;
    e->exporting = true;
    e->done = (c.active == 0);
    e->dev_seconds = 0.0;
    return PBB_OK;
}

int pbb_get_intervals(pbb_engine* e, int32_t max_intervals, int32_t* pos, int32_t* end, int32_t* ids,
                      int32_t* nb_intervals)
{
    if (!e || !e->started) return fail(PBB_E_INVAL, "engine not started");
    if (!nb_intervals) return fail(PBB_E_INVAL, "nb_intervals is NULL");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(cudaStreamSynchronize(e->st));
    e->exporting = true;
    const int B = e->cfg.nb_ivms, n = e->H.n, npad = e->npad;
    std::vector<int> st(B);
    std::vector<signed char> ps((size_t)B * npad), es((size_t)B * npad);
    CK(cudaMemcpy(st.data(), e->state, sizeof(int) * B, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(ps.data(), e->group.ivm.pos, ps.size(), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(es.data(), e->group.ivm.end, es.size(), cudaMemcpyDeviceToHost));
    // An explorer stopped between selection steps may hold a digit one past
    // its level's last cell (n - l: "this level is done"); carry it into the
    // level above (ivm::goUp, multicore/src/ivm.cpp:56-72) so that every
    // exported digit lies in [0, n - l), and drop intervals the carry empties.
    std::vector<int> keep;
    std::vector<int> pv((size_t)B * n), ev((size_t)B * n);
    for (int k = 0; k < B; k++) {
        if (st[k] != IVM_ACTIVE) continue;
        int* a = &pv[(size_t)k * n];
        int* z = &ev[(size_t)k * n];
        for (int i = 0; i < n; i++) {
            a[i] = ps[(size_t)k * npad + i];
            z[i] = es[(size_t)k * npad + i];
        }
        for (int l = n - 1; l > 0; l--)
            if (a[l] >= n - l) { a[l] = 0; a[l - 1]++; }
        if (a[0] >= n) continue;
        bool le = true;     // pos <= end, lexicographically
        for (int l = 0; l < n; l++)
            if (a[l] != z[l]) { le = a[l] < z[l]; break; }
        if (le) keep.push_back(k);
    }
    const int cnt = (int)keep.size();
    *nb_intervals = cnt;
    if (cnt > max_intervals) return fail(PBB_E_INVAL, "buffer too small for the active intervals");
    if (cnt > 0 && (!pos || !end)) return fail(PBB_E_INVAL, "pos/end are NULL");
    for (int w = 0; w < cnt; w++) {
        const int k = keep[w];
        for (int i = 0; i < n; i++) {
            pos[(size_t)w * n + i] = pv[(size_t)k * n + i];
            end[(size_t)w * n + i] = ev[(size_t)k * n + i];
        }
        if (ids) ids[w] = k;
    }
    return PBB_OK;
}

int pbb_set_ub(pbb_engine* e, int32_t ub)
{
    if (!e || !e->started) return fail(PBB_E_INVAL, "engine not started");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(pbbl::launch_lower_ub(e->group_d, 0, ub, e->st));
    CK(cudaStreamSynchronize(e->st));
    return PBB_OK;
}

int pbb_set_wait_limit(pbb_engine* e, double seconds)
{
    if (!e) return fail(PBB_E_INVAL, "engine is NULL");
    e->wait_limit_s = seconds;
    return PBB_OK;
}

int pbb_diag_set_step_limits(pbb_engine* e, int32_t select_budget, int32_t max_rounds)
{
    if (!e) return fail(PBB_E_INVAL, "engine is NULL");
    if (select_budget < 1 || max_rounds < 1) return fail(PBB_E_INVAL, "limits must be >= 1");
    e->select_budget = select_budget;
    e->max_rounds = max_rounds;
    return PBB_OK;
}

static int sample_nodes(pbb_engine* e, int32_t capacity, int32_t rate_log2, bool decisions)
{
    if (!e) return fail(PBB_E_INVAL, "engine is NULL");
    if (decisions && (e->pair_warps <= 0 || !PBB_VAR_PAIRS(e->pair_variant)))
        return fail(PBB_E_UNSUPPORTED, "this search does not run with kept pair bounds");
    if (capacity < 0 || rate_log2 < 0 || rate_log2 > 30) return fail(PBB_E_INVAL, "bad sampling parameters");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(cudaStreamSynchronize(e->st));
    pbbh::mem_free(e->sample_d, e->lease);
    pbbh::mem_free(e->sample_rec, e->lease);
    e->sample_d = nullptr;
    e->sample_rec = nullptr;
    e->group.sample = nullptr;
    e->sample_decisions = decisions;
    if (capacity > 0) {
        e->sample_stride = PBB_SAMPLE_HDR + 5 * e->H.n;
        const size_t bytes = sizeof(int) * (size_t)capacity * e->sample_stride;
        CK(pbbh::mem_alloc((void**)&e->sample_rec, bytes, e->lease));
        CK(pbbh::mem_alloc((void**)&e->sample_d, sizeof(SampleBuf), e->lease));
        CK(cudaMemsetAsync(e->sample_rec, 0, bytes, e->st));
        SampleBuf sb;
        sb.count = 0;
        sb.cap = (unsigned)capacity;
        sb.rate_mask = (1u << rate_log2) - 1u;
        sb.stride = e->sample_stride;
        sb.rec = e->sample_rec;
        CK(cudaMemcpyAsync(e->sample_d, &sb, sizeof(sb), cudaMemcpyHostToDevice, e->st));
        e->group.sample = e->sample_d;
    }
    CK(cudaMemcpyAsync(e->group_d, &e->group, sizeof(DevGroup), cudaMemcpyHostToDevice, e->st));
    CK(cudaStreamSynchronize(e->st));
    return PBB_OK;
}

int pbb_diag_sample_nodes(pbb_engine* e, int32_t capacity, int32_t rate_log2)
{
    return sample_nodes(e, capacity, rate_log2, false);
}

int pbb_diag_sample_decisions(pbb_engine* e, int32_t capacity, int32_t rate_log2)
{
    return sample_nodes(e, capacity, rate_log2, true);
}

int pbb_diag_get_samples(pbb_engine* e, int32_t max_records, int32_t* out, int32_t* count)
{
    if (!e || !count) return fail(PBB_E_INVAL, "NULL argument");
    *count = 0;
    if (!e->sample_d) return PBB_OK;
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(cudaStreamSynchronize(e->st));
    SampleBuf sb;
    CK(cudaMemcpy(&sb, e->sample_d, sizeof(sb), cudaMemcpyDeviceToHost));
    const int have = (int)std::min(sb.count, sb.cap);
    const int k = std::min(have, std::max(0, (int)max_records));
    if (k > 0) {
        if (!out) return fail(PBB_E_INVAL, "out is NULL");
        CK(cudaMemcpy(out, e->sample_rec, sizeof(int) * (size_t)k * e->sample_stride, cudaMemcpyDeviceToHost));
    }
    *count = max_records > 0 ? k : have;
    return PBB_OK;
}

static int explore_window(pbb_engine* e, double seconds, int32_t* done, int eager)
{
    if (!e || !e->started) return fail(PBB_E_INVAL, "engine not started");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    int rc = settle(e);
    if (rc) return rc;
    if (!e->done) {
        // a launch never runs unbounded: at most 120 s of device time per window
        const double win = (seconds > 0 && seconds < 120.0) ? seconds : 120.0;
        const unsigned long long budget = (unsigned long long)(win * 1e9);
        CK(cudaEventRecord(e->ev0, e->st));
        int variant = (e->cfg.sorted_dfs || e->cfg.early_stop_johnson) ? 1 : 0;
        if (e->pair_warps > 0) variant = e->pair_variant;
        // sampling: by the search's own build, but for the Johnson values of a
        // search with kept pair bounds, which computes none
        if (e->sample_d) {
            if (variant == 7) variant = 10;
            else if (e->sample_decisions) variant = PBB_VAR_GEN(variant) ? 9 : 8;
            else variant = 2;
        }
        const bool own = variant >= 3;
        const int warps = std::min(own ? e->pair_warps : e->warps, PBB_EXPLORE_WARPS(variant));
        CK(pbbl::launch_explore(e->nw, e->group_d, e->ngroups_d, e->ctas, warps, own ? e->pair_smem : e->smem, budget,
                                e->max_rounds, e->select_budget, e->st,
                                variant, eager, e->pair_stack, e->pair_stride));
        CK(cudaEventRecord(e->ev1, e->st));
        rc = wait_event(e->ev1, e->wait_limit_s < 0 ? win + 60.0 : e->wait_limit_s);
        if (rc == PBB_E_TIMEOUT) {
            e->pending = true;
            return fail(PBB_E_TIMEOUT, "the exploration window did not end within the host wait limit; it ends by "
                                       "its own device-time budget and the next call accounts for it");
        }
        if (rc) return rc;
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, e->ev0, e->ev1));
        e->dev_seconds += ms * 1e-3;
        int active = 0;
        CK(cudaMemcpy(&active, &e->ctl->active, sizeof(int), cudaMemcpyDeviceToHost));
        e->done = (active == 0);
    }
    if (done) *done = e->done ? 1 : 0;
    return PBB_OK;
}

// A caller that exports intervals between windows pays for every one: the
// engine that resumes it bounds its path again.  So the first window of a
// search, and one after an export, keeps to share_after when it is shorter than
// this, and a caller that comes back without having exported gets eager windows
// from then on.  Intervals after a first window kept to share_after / an eager
// one: 2 ms 20x20 15 / 2924, 16x20 16 / 2914, 24x10 84 / done; 5 ms 330 / 4700,
// 383 / 2803, 552 / done; at 9 ms 2935 / 4692 and 2899 / done, not worth the
// speed: device ms of whole searches 20x20 42 / 32, 16x20 14.4 / 6.1, 24x10
// 10 / 1.6, 13x20 8.5 / 0.9.
#define PBB_SHORT_WINDOW_S 0.005

int pbb_explore(pbb_engine* e, double seconds, int32_t* done)
{
    if (!e || !e->started) return fail(PBB_E_INVAL, "engine not started");
    const bool may_export = e->exporting && seconds > 0 && seconds < PBB_SHORT_WINDOW_S;
    e->exporting = false;
    return explore_window(e, seconds, done, !may_export);
}

int pbb_get_result(pbb_engine* e, pbb_result* out)
{
    if (!e || !out) return fail(PBB_E_INVAL, "NULL argument");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(cudaStreamSynchronize(e->st));
    GroupCtl c;
    CK(cudaMemcpy(&c, e->ctl, sizeof(c), cudaMemcpyDeviceToHost));
    memset(out, 0, sizeof(*out));
    out->complete = e->done ? 1 : 0;
    const unsigned best_id = (unsigned)(c.best_key & 0xffffffffull);
    // a bound lowered from outside (pbb_set_ub) carries no permutation here
    out->found = (c.found > 0 && best_id != 0xffffffffu) ? 1 : 0;
    out->cost = (int32_t)(c.best_key >> 32);
    out->n_jobs = e->H.n;
    out->stats.decomposed = c.decomposed;
    out->stats.johnson_bounds = c.johnson_bounds;
    out->stats.simple_bounds = c.simple_bounds;
    out->stats.leaves = c.leaves;
    out->stats.steals = c.steals;
    out->device_seconds = e->dev_seconds;
    if (c.status & PBB_ST_BADINPUT) return fail(PBB_E_INVAL, "device reported bad input");
    if (out->found) {
        const unsigned id = (unsigned)(c.best_key & 0xffffffffull);
        if (id >= (unsigned)e->cfg.nb_ivms) return fail(PBB_E_CUDA, "corrupt best key");
        signed char buf[PBB_MAX_N];
        CK(cudaMemcpy(buf, e->bestperm + (size_t)id * e->npad, e->H.n, cudaMemcpyDeviceToHost));
        for (int i = 0; i < e->H.n; i++) out->perm[i] = buf[i];
        out->has_perm = 1;
    } else if (e->from_neh && out->cost == e->ub) {
        // not improved: the NEH schedule the search started from
        int buf[PBB_MAX_N + 1];
        CK(cudaMemcpy(buf, e->neh_d, sizeof(buf), cudaMemcpyDeviceToHost));
        for (int i = 0; i < e->H.n; i++) out->perm[i] = buf[i];
        out->has_perm = 1;
    } else if ((int)e->start_perm.size() == e->H.n && out->cost == e->ub) {
        // not improved: the schedule that came with the starting bound
        for (int i = 0; i < e->H.n; i++) out->perm[i] = e->start_perm[i];
        out->has_perm = 1;
    }
    return PBB_OK;
}

int pbb_solve(pbb_engine* e, int32_t ub, const int32_t* root_perm, double time_limit_s, pbb_result* out)
{
    int rc = pbb_start(e, ub, root_perm);
    if (rc) return rc;
    int32_t done = e->done ? 1 : 0;
    while (!done) {
        double slice = e->slice_s;
        if (time_limit_s > 0) {
            const double left = time_limit_s - e->dev_seconds;
            if (left <= 0) break;
            slice = std::min(slice, left);
        }
        rc = explore_window(e, slice, &done, 1);
        if (rc) return rc;
    }
    return pbb_get_result(e, out);
}

static int bound_children_impl(const pbb_instance* inst, int32_t johnson_mode, int32_t device, int32_t method,
                               int32_t count, const int32_t* sched, const int32_t* limit1, const int32_t* limit2,
                               int32_t* weak_begin, int32_t* weak_end, int32_t* strong_begin, int32_t* strong_end,
                               int32_t* node_weak, int32_t* node_strong, int32_t* prio_begin = nullptr,
                               int32_t* prio_end = nullptr, int32_t* strong_idle = nullptr);

int pbb_bound_children(const pbb_instance* inst, int32_t johnson_mode, int32_t device, int32_t count,
                       const int32_t* sched, const int32_t* limit1, const int32_t* limit2, int32_t* weak_begin,
                       int32_t* weak_end, int32_t* strong_begin, int32_t* strong_end, int32_t* node_weak,
                       int32_t* node_strong)
{
    return bound_children_impl(inst, johnson_mode, device, -1, count, sched, limit1, limit2, weak_begin, weak_end,
                               strong_begin, strong_end, node_weak, node_strong);
}

int pbb_bound_children_ex(const pbb_instance* inst, int32_t johnson_mode, int32_t device, int32_t count,
                          const int32_t* sched, const int32_t* limit1, const int32_t* limit2, const pbb_bound_out* out)
{
    if (!out) return fail(PBB_E_INVAL, "out is NULL");
    return bound_children_impl(inst, johnson_mode, device, -1, count, sched, limit1, limit2, out->weak_begin,
                               out->weak_end, out->strong_begin, out->strong_end, out->node_weak, out->node_strong,
                               out->prio_begin, out->prio_end, out->strong_idle);
}

int pbb_diag_bound_children(const pbb_instance* inst, int32_t johnson_mode, int32_t device, int32_t method,
                            int32_t count, const int32_t* sched, const int32_t* limit1, const int32_t* limit2,
                            int32_t* weak_begin, int32_t* weak_end, int32_t* strong_begin, int32_t* strong_end,
                            int32_t* node_weak, int32_t* node_strong)
{
    if (method < 0 || method > 2)
        return fail(PBB_E_INVAL, "method must be 0 (sweeps), 1 (direct scans) or 2 (sweeps over free positions)");
    return bound_children_impl(inst, johnson_mode, device, method, count, sched, limit1, limit2, weak_begin,
                               weak_end, strong_begin, strong_end, node_weak, node_strong);
}

static int bound_children_impl(const pbb_instance* inst, int32_t johnson_mode, int32_t device, int32_t method,
                               int32_t count, const int32_t* sched, const int32_t* limit1, const int32_t* limit2,
                               int32_t* weak_begin, int32_t* weak_end, int32_t* strong_begin, int32_t* strong_end,
                               int32_t* node_weak, int32_t* node_strong, int32_t* prio_begin, int32_t* prio_end,
                               int32_t* strong_idle)
{
    if (count < 0 || (count > 0 && (!sched || !limit1 || !limit2))) return fail(PBB_E_INVAL, "bad node arrays");
    HostTables H;
    int rc = build_tables(inst, johnson_mode, H);
    if (rc) return rc;
    if (count == 0) return PBB_OK;
    const int n = H.n;
    for (int i = 0; i < count; i++) {
        if (limit1[i] < -1 || limit2[i] > n || limit1[i] >= limit2[i]) return fail(PBB_E_INVAL, "bad limits");
        unsigned long long seen = 0ull;
        for (int t = 0; t < n; t++) {
            const int j = sched[(size_t)i * n + t];
            if (j < 0 || j >= n || ((seen >> j) & 1ull)) return fail(PBB_E_INVAL, "schedule is not a permutation");
            seen |= 1ull << j;
        }
    }
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(device));
    pbbh::Lease lease;
    CK(pbbh::stream_take(&lease, device));
    const cudaStream_t st = lease.st;
    const size_t cn = (size_t)count * n * sizeof(int), c1 = (size_t)count * sizeof(int);
    const bool want_prio = prio_begin || prio_end;
    // one block: tables, status and inputs, then the outputs.  Up to
    // PACKED_BYTES of inputs go up in one copy with the tables, and as many of
    // outputs come back in one.
    const size_t PACKED_BYTES = 256 * 1024;
    pbbh::Carver C;
    const InstanceBlock tables(H, C);
    const size_t o_status = C.take(sizeof(unsigned));
    const size_t o_tables_end = C.bytes;
    const size_t o_s = C.take(cn), o_l1 = C.take(c1), o_l2 = C.take(c1);
    const size_t o_inputs_end = C.bytes;
    struct Out { int32_t* host; size_t off, bytes; };
    Out out[9] = {{weak_begin, 0, cn}, {weak_end, 0, cn}, {strong_begin, 0, cn}, {strong_end, 0, cn},
                  {node_weak, 0, c1}, {node_strong, 0, c1}, {prio_begin, 0, cn}, {prio_end, 0, cn},
                  {strong_idle, 0, c1}};
    for (int q = 0; q < 9; q++)
        if (q < 6 || (q < 8 && want_prio) || (q == 8 && strong_idle)) out[q].off = C.take(out[q].bytes);
    unsigned char* d = nullptr;
    do {
        cudaError_t ce = pbbh::mem_alloc((void**)&d, C.bytes, lease);
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "cudaMalloc"); break; }
        const bool packed_in = o_inputs_end - o_tables_end <= PACKED_BYTES;
        std::vector<unsigned char> host(packed_in ? o_inputs_end : o_tables_end, 0);
        tables.fill(H, host.data());
        if (packed_in) {
            memcpy(host.data() + o_s, sched, cn);
            memcpy(host.data() + o_l1, limit1, c1);
            memcpy(host.data() + o_l2, limit2, c1);
        } else {
            ce = cudaMemcpyAsync(d + o_s, sched, cn, cudaMemcpyHostToDevice, st);
            if (!ce) ce = cudaMemcpyAsync(d + o_l1, limit1, c1, cudaMemcpyHostToDevice, st);
            if (!ce) ce = cudaMemcpyAsync(d + o_l2, limit2, c1, cudaMemcpyHostToDevice, st);
        }
        if (!ce) ce = cudaMemcpyAsync(d, host.data(), host.size(), cudaMemcpyHostToDevice, st);
        int sms = 0;
        if (!ce) ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "upload of the tables and nodes"); break; }
        const pbbl::BoundShape shape = pbbl::bound_shape(n, H.m, H.Ppad, count, sms, max_smem_optin(device));
        if (shape.warps < 1) { rc = fail(PBB_E_INVAL, "instance tables do not fit in shared memory"); break; }
        auto dev = [&](size_t off) { return reinterpret_cast<int*>(d + off); };
        BoundExtra X;
        if (want_prio) { X.prio_begin = dev(out[6].off); X.prio_end = dev(out[7].off); }
        if (strong_idle) X.strong_idle = dev(out[8].off);
        unsigned* status = reinterpret_cast<unsigned*>(d + o_status);
        const int nw = n <= 32 ? 1 : 2;
        if (method < 0) {
            ce = pbbl::launch_bound_all(nw, tables.view(H, d), count, dev(o_s), dev(o_l1), dev(o_l2), dev(out[0].off),
                                        dev(out[1].off), dev(out[2].off), dev(out[3].off), dev(out[4].off),
                                        dev(out[5].off), status, shape, st, X);
        } else {
            int smem = 0;
            const int warps = pick_warps(H, 8, device, smem);
            const int ctas = std::min((count + warps - 1) / warps, sms * 4);
            ce = pbbl::launch_bound(nw, tables.view(H, d), count, dev(o_s), dev(o_l1), dev(o_l2), dev(out[0].off),
                                    dev(out[1].off), dev(out[2].off), dev(out[3].off), dev(out[4].off),
                                    dev(out[5].off), status, ctas, warps, smem, st, method, X);
        }
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "pbb_bound_kernel launch"); break; }
        unsigned hs = 0;
        ce = cudaMemcpyAsync(&hs, status, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
        const size_t back = C.bytes - o_inputs_end;
        std::vector<unsigned char> packed(back <= PACKED_BYTES ? back : 0);
        if (!packed.empty()) {
            if (!ce) ce = cudaMemcpyAsync(packed.data(), d + o_inputs_end, back, cudaMemcpyDeviceToHost, st);
        } else {
            for (const Out& o : out)
                if (!ce && o.host && o.off) ce = cudaMemcpyAsync(o.host, d + o.off, o.bytes, cudaMemcpyDeviceToHost, st);
        }
        // the copies under way read and write this frame's buffers
        const cudaError_t end = cudaStreamSynchronize(st);
        if (!ce) ce = end;
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "pbb_bound_kernel"); break; }
        if (hs & PBB_ST_BADINPUT) { rc = fail(PBB_E_INVAL, "device rejected a node"); break; }
        if (!packed.empty())
            for (const Out& o : out)
                if (o.host && o.off) memcpy(o.host, packed.data() + (o.off - o_inputs_end), o.bytes);
    } while (0);
    cudaStreamSynchronize(st);
    pbbh::mem_free(d, lease);
    pbbh::stream_give(lease);
    return rc;
}

int pbb_work_counters(pbb_engine* e, pbb_work* out)
{
    if (!e || !out) return fail(PBB_E_INVAL, "NULL argument");
    pbbh::DeviceGuard keep_callers_device;
    CK(cudaSetDevice(e->dev));
    {
        const int rs = settle(e);
        if (rs) return rs;
    }
    CK(cudaStreamSynchronize(e->st));
    GroupCtl c;
    CK(cudaMemcpy(&c, e->ctl, sizeof(c), cudaMemcpyDeviceToHost));
    out->device_seconds = e->dev_seconds;
    out->n_jobs = e->H.n;
    out->n_machines = e->H.m;
    out->machine_pairs = e->H.P;
    out->decomposed = c.decomposed;
    out->simple_bounds = c.simple_bounds;
    out->johnson_bounds = c.johnson_bounds;
    out->johnson_sweeps = c.jsweeps;
    out->sweep_free_jobs = c.jfree;
    out->sweep_children = c.jchild;
    out->direct_children = c.jdirect;
    out->direct_free_jobs = e->H.P > 0 ? c.jdirect_free / e->H.P : 0;   // counted over the machine pairs
    out->explorers = e->cfg.nb_ivms;
    out->warps = (e->pair_warps > 0 ? e->pair_warps : e->warps) * e->ctas;
    out->status = (int32_t)c.status;
    return PBB_OK;
}

// NEH (heuristic/src/fastNEH.cpp:230-243 for the insertion procedure): jobs
// by decreasing total time (ties: lower id first); the first two keep the
// swapped order unless the original one is strictly better; each next job is
// inserted at the first position of least partial makespan.
int pbb_neh(const pbb_instance* inst, int32_t* perm, int32_t* cost)
{
    if (!inst || !inst->p || !perm) return fail(PBB_E_INVAL, "NULL argument");
    const int n = inst->n_jobs, m = inst->n_machines;
    if (n < 1 || m < 1) return fail(PBB_E_INVAL, "empty instance");
    const int32_t* p = inst->p;
    std::vector<int> tot(n, 0), order(n);
    for (int j = 0; j < n; j++) {
        for (int k = 0; k < m; k++) tot[j] += p[k * n + j];
        order[j] = j;
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tot[a] > tot[b]; });
    std::vector<int> c(m);
    auto makespan = [&](const std::vector<int>& s) {
        std::fill(c.begin(), c.end(), 0);
        for (int j : s) {
            c[0] += p[j];
            for (int k = 1; k < m; k++) c[k] = std::max(c[k - 1], c[k]) + p[k * n + j];
        }
        return c[m - 1];
    };
    std::vector<int> seq;
    if (n == 1) {
        seq = {order[0]};
    } else {
        std::vector<int> a = {order[0], order[1]}, b = {order[1], order[0]};
        seq = makespan(a) < makespan(b) ? a : b;
        for (int k = 2; k < n; k++) {
            int best = INT_MAX, bpos = 0;
            std::vector<int> trial;
            for (int q = 0; q <= k; q++) {
                trial = seq;
                trial.insert(trial.begin() + q, order[k]);
                const int v = makespan(trial);
                if (v < best) { best = v; bpos = q; }
            }
            seq.insert(seq.begin() + bpos, order[k]);
        }
    }
    for (int i = 0; i < n; i++) perm[i] = seq[i];
    if (cost) *cost = makespan(seq);
    return PBB_OK;
}

}  // extern "C"
