// Initial upper bounds on the device: NEH (heuristic/src/fastNEH.cpp:230-243
// for the insertion procedure), one warp per instance, and iterated greedy,
// eight warps per instance, for many instances in one launch -- the pool
// computes its admissions' bounds this way, without a host round trip, and the
// engine can start from it.
//
// Insertion of job x into a sequence of `len` jobs uses Taillard's heads and
// tails (fastNEH.cpp:100-178 computeHeads / computeTails / insertJob /
// findBestPos restated): with e the heads of the sequence and q its tails,
// inserting x at position i gives the makespan
//   max_k ( f_k + q_i,k ),  f_k = max(f_{k-1}, e_{i-1,k}) + p_k(x),
// exactly the makespan of the sequence with x at i.  Heads and tails run as
// one diagonal wavefront (one machine per lane), the insertion costs one
// position per lane.  Integer only: the result equals the host restatement
// pbb_neh job for job.
//
// What bounds these kernels is the serial chain of one instance, not the GPU's
// throughput: a wavefront step is one shuffle, one max and one add for every
// machine, where a max-plus scan per job took ten shuffles (NEH of 64
// instances of 50 x 20, whole call with 0.9 ms of host work: 1.9 -> 1.25 ms).
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "pbb_types.h"
#include "pbb_heur.h"
#include "pbb_devguard.h"
#include "pbb_mem.h"
#include "pbb_tables.h"
#include "../../include/pbbperm.h"

namespace {

#define HEUR_FULL 0xffffffffu

__device__ __forceinline__ int hlane() { return threadIdx.x & 31; }

// Heads of `la` jobs appended to a sequence whose heads are h0 (job r:
// ahead[r]), and tails of `lb` jobs put before one whose tails are t0 (job r:
// behind[-r]), lane = machine, as one wavefront; row r of the results at
// E + r * PBB_HEUR_ROW and Q + r * qstep.  m lanes used.
__device__ __forceinline__ void wavefront(const int* pt, int mp, int m, int h0, const int* ahead, int la, int* E,
                                          int t0, const int* behind, int lb, int* Q, int qstep)
{
    const int lane = hlane();
    const int steps = max(la, lb) + m - 1;
    const int back = m - 1 - lane;         // the last machine leads the tails
    int cf = h0, cb = t0;
    for (int s = 0; s < steps; s++) {
        int up = __shfl_up_sync(HEUR_FULL, cf, 1), dn = __shfl_down_sync(HEUR_FULL, cb, 1);
        if (lane == 0) up = 0;
        if (lane == m - 1) dn = 0;
        const int i = s - lane, j = s - back;
        if (lane < m && i >= 0 && i < la) {
            cf = max(cf, up) + pt[ahead[i] * mp + lane];
            E[i * PBB_HEUR_ROW + lane] = cf;
        }
        if (lane < m && j >= 0 && j < lb) {
            cb = max(cb, dn) + pt[behind[-j] * mp + lane];
            Q[j * qstep + lane] = cb;
        }
    }
}

// Heads E[i] (positions 0..len-1) and tails Q[i] (0..len, Q[len] = 0) of
// seq[0..len), one machine per lane, stored by position.
__device__ __forceinline__ void heads_tails(const int* pt, int mp, int m, const int* seq, int len, int* E, int* Q)
{
    Q[len * PBB_HEUR_ROW + hlane()] = 0;
    wavefront(pt, mp, m, 0, seq, len, E, 0, seq + len - 1, len, Q + (len - 1) * PBB_HEUR_ROW, -PBB_HEUR_ROW);
    __syncwarp();
}

// makespan of jobs a then b, read by every lane
__device__ __forceinline__ int pair_makespan(const int* pt, int mp, int m, int a, int b)
{
    int h1 = 0, h2 = 0;
    for (int k = 0; k < m; k++) {
        h1 += pt[a * mp + k];
        h2 = max(h1, h2) + pt[b * mp + k];
    }
    return h2;
}

// makespan of job x between the heads e (NULL: none) and the tails q
__device__ __forceinline__ int insert_cost(const int* pt, int mp, int m, const int* e, const int* q, int x)
{
    const int* px = pt + x * mp;
    int f = 0, c = 0;
#pragma unroll 4
    for (int k = 0; k < m; k++) {
        f = max(f, e ? e[k] : 0) + px[k];
        c = max(c, f + q[k]);
    }
    return c;
}

// smallest (makespan << 32) | position over the lanes
__device__ __forceinline__ unsigned long long least_key(unsigned long long best)
{
    const unsigned hi = __reduce_min_sync(HEUR_FULL, (unsigned)(best >> 32));
    const unsigned lo = __reduce_min_sync(HEUR_FULL, (unsigned)(best >> 32) == hi ? (unsigned)best : 0xffffffffu);
    return ((unsigned long long)hi << 32) | lo;
}

// Makespan of x inserted at the best position of the sequence of `len` jobs
// whose heads and tails are E, Q (fastNEH.cpp:120-178): the first position
// of least makespan.  Returns (makespan << 32) | position, on every lane.
__device__ __forceinline__ unsigned long long best_insert(const int* pt, int mp, int m, const int* E, const int* Q,
                                                          int x, int len)
{
    unsigned long long best = ~0ull;
    for (int i = hlane(); i <= len; i += 32) {
        const int c = insert_cost(pt, mp, m, i > 0 ? E + (i - 1) * PBB_HEUR_ROW : nullptr, Q + i * PBB_HEUR_ROW, x);
        const unsigned long long key = ((unsigned long long)(unsigned)c << 32) | (unsigned)i;
        best = key < best ? key : best;
    }
    return least_key(best);
}

// The same for the job at position i of the whole sequence seq[0..n), taken
// out and put back within `reach` places; E, Q: heads and tails of the whole
// sequence.  Without the job, heads before i and tails behind it stay as they
// are, so only the rows between i and the reach are computed, into Er and Qr:
// a probe costs 2 x reach jobs instead of two passes over the sequence.
__device__ __forceinline__ unsigned long long probe_move(const int* pt, int mp, int n, int m, const int* seq,
                                                         const int* E, const int* Q, int i, int reach, int* Er, int* Qr)
{
    const int lane = hlane();
    const int lo = max(0, i - reach), hi = min(n - 1, i + reach);
    const int h0 = i > 0 && lane < m ? E[(i - 1) * PBB_HEUR_ROW + lane] : 0;
    const int t0 = lane < m ? Q[(i + 1) * PBB_HEUR_ROW + lane] : 0;
    __syncwarp();
    wavefront(pt, mp, m, h0, seq + i + 1, hi - i, Er, t0, seq + i - 1, i - lo, Qr, PBB_HEUR_ROW);
    __syncwarp();
    unsigned long long best = ~0ull;
    const int q = lo + lane;               // at most 2 x 8 + 1 positions
    if (q <= hi) {
        const int* e = q == 0 ? nullptr : (q - 1 < i ? E + (q - 1) * PBB_HEUR_ROW : Er + (q - 1 - i) * PBB_HEUR_ROW);
        const int* t = q >= i ? Q + (q + 1) * PBB_HEUR_ROW : Qr + (i - 1 - q) * PBB_HEUR_ROW;
        best = ((unsigned long long)(unsigned)insert_cost(pt, mp, m, e, t, seq[i]) << 32) | (unsigned)q;
    }
    return least_key(best);
}

// seq[0..len) -> seq[0..len] with x at position pos
__device__ __forceinline__ void insert_at(int* seq, int len, int pos, int x)
{
    const int lane = hlane();
    int moved[2];
    for (int w = 0; w < 2; w++) {
        const int i = w * 32 + lane;
        moved[w] = (i >= pos && i < len) ? seq[i] : -1;
    }
    __syncwarp();
    for (int w = 0; w < 2; w++) {
        const int i = w * 32 + lane;
        if (moved[w] >= 0) seq[i + 1] = moved[w];
    }
    if (lane == 0) seq[pos] = x;
    __syncwarp();
}

// seq[0..len) -> seq[0..len-1) without position pos; returns the job removed
__device__ __forceinline__ int remove_at(int* seq, int len, int pos)
{
    const int lane = hlane();
    const int x = seq[pos];
    int moved[2];
    for (int w = 0; w < 2; w++) {
        const int i = w * 32 + lane;
        moved[w] = (i > pos && i < len) ? seq[i] : -1;
    }
    __syncwarp();
    for (int w = 0; w < 2; w++) {
        const int i = w * 32 + lane;
        if (moved[w] >= 0) seq[i - 1] = moved[w];
    }
    __syncwarp();
    return x;
}

struct HeurSmem {
    int *pt, *E, *Q, *seq, *order, *tot, *cur, *best, *vo, *probe;
    int mp;                                     // row stride of pt
};

__device__ __forceinline__ HeurSmem heur_smem(int* hs, int m)
{
    HeurSmem S;
    S.pt = hs;                                  // [n][mp]
    S.E = S.pt + PBB_MAX_N * 36;                // [PBB_MAX_N] rows: heads by position
    S.Q = S.E + PBB_MAX_N * PBB_HEUR_ROW;       // [PBB_MAX_N + 1] rows: tails by position
    S.seq = S.Q + (PBB_MAX_N + 1) * PBB_HEUR_ROW;   // [PBB_MAX_N] each of the following
    S.order = S.seq + PBB_MAX_N;
    S.tot = S.order + PBB_MAX_N;
    S.cur = S.tot + PBB_MAX_N;
    S.best = S.cur + PBB_MAX_N;
    S.vo = S.best + PBB_MAX_N;
    S.probe = S.vo + PBB_MAX_N;                 // iterated greedy: two sets of rows per warp
    S.mp = pbb_machine_pad(m);
    return S;
}

// the instance's times, job by job
__device__ __forceinline__ void load_times(const HeurSmem& S, const int* p, int n, int m)
{
    for (int i = threadIdx.x; i < n * m; i += blockDim.x) {
        const int k = i / n, j = i - k * n;
        S.pt[j * S.mp + k] = p[i];
    }
}

// NEH into S.seq; returns the makespan (every lane)
__device__ int neh_warp(const HeurSmem& S, int n, int m)
{
    const int lane = hlane();
    const int* pt = S.pt;
    const int mp = S.mp;
    // total time per job, then the jobs by decreasing total (ties: lower id first)
    for (int j = lane; j < n; j += 32) {
        int s = 0;
        for (int k = 0; k < m; k++) s += pt[j * mp + k];
        S.tot[j] = s;
    }
    __syncwarp();
    for (int j = lane; j < n; j += 32) {
        int r = 0;
        for (int i = 0; i < n; i++) r += (S.tot[i] > S.tot[j] || (S.tot[i] == S.tot[j] && i < j)) ? 1 : 0;
        S.order[r] = j;
    }
    __syncwarp();
    if (n == 1) {
        if (lane == 0) S.seq[0] = S.order[0];
        __syncwarp();
        return S.tot[0];
    }
    // the first two keep the swapped order unless the original one is
    // strictly better (fastNEH.cpp:233-236)
    const int a = S.order[0], b = S.order[1];
    const int ca = pair_makespan(pt, mp, m, a, b), cb = pair_makespan(pt, mp, m, b, a);
    if (lane == 0) {
        S.seq[0] = ca < cb ? a : b;
        S.seq[1] = ca < cb ? b : a;
    }
    __syncwarp();
    int cost = min(ca, cb);
    for (int len = 2; len < n; len++) {
        const int x = S.order[len];
        heads_tails(pt, mp, m, S.seq, len, S.E, S.Q);
        const unsigned long long key = best_insert(pt, mp, m, S.E, S.Q, x, len);
        insert_at(S.seq, len, (int)(key & 0xffffffffu), x);
        cost = (int)(key >> 32);
    }
    return cost;
}

// splitmix64 step (the project's generator), lane 0 only
__device__ __forceinline__ unsigned long long rng_next(unsigned long long& s)
{
    s += 0x9E3779B97F4A7C15ull;
    unsigned long long z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// uniform integer in [a, b] from the high word of a 64x(b-a+1) product
__device__ __forceinline__ int rng_range(unsigned long long& s, int a, int b)
{
    return a + (int)__umul64hi(rng_next(s), (unsigned long long)(b - a + 1));
}

}  // namespace

// One warp per task.  Dynamic shared memory: PBB_HEUR_SMEM bytes.
__global__ void __launch_bounds__(32) pbb_neh_kernel(const NehTask* tasks, int count)
{
    extern __shared__ __align__(16) int hs[];
    const int t = blockIdx.x;
    if (t >= count) return;
    const NehTask T = tasks[t];
    const int n = T.n, m = T.m, lane = hlane();
    const HeurSmem S = heur_smem(hs, m);
    load_times(S, T.p, n, m);
    __syncwarp();
    const int cost = neh_warp(S, n, m);
    for (int i = lane; i < n; i += 32) T.perm[i] = S.seq[i];
    if (lane == 0) {
        if (T.cost) *T.cost = cost;
        if (T.ub) *T.ub = cost;
    }
}

// Iterated greedy from the NEH schedule (heuristic/src/IG.cpp:341-416 runIG,
// destruction :120-160, construction :229-255, localSearchKI :567-612,
// acceptance :258-274), one block per task.  Every random decision is drawn by
// thread 0 from the task's splitmix64 stream (seed + task index), in this
// order per round: the destruction's window r, its shuffle, then the
// acceptance draw; a worse schedule is kept with probability T / (T + delta),
// T = 0.2 x mean processing time / 10 (the reference's temperature, with the
// exponential replaced by a rational of the same shape so that the test is
// integer arithmetic).  The host restatement in the test oracle follows the
// same stream.
//
// The local search takes nearly all of the time: a probe per job, the first
// improvement taken.  The block's warps probe the next jobs of the visit order
// at once, and the first in that order that improves is taken, which is the
// one a single warp would have come to; a pass computes the whole sequence's
// heads and tails once for all its probes.  64 instances of 50 x 20, five
// rounds, whole call: 23.7 ms with one warp and two whole passes per probe,
// 2.4 ms so (NEH alone 1.2).
__global__ void __launch_bounds__(32 * PBB_IG_WARPS) pbb_ig_kernel(const NehTask* tasks, int count, IgParams prm)
{
    extern __shared__ __align__(16) int hs[];
    const int t = blockIdx.x;
    if (t >= count) return;
    const NehTask T = tasks[t];
    const int n = T.n, m = T.m, lane = hlane();
    const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const HeurSmem S = heur_smem(hs, m);
    __shared__ int removed[PBB_MAX_N];
    __shared__ unsigned long long found[PBB_IG_WARPS];
    __shared__ int sh_cost, sh_accept;
    load_times(S, T.p, n, m);
    __syncthreads();
    if (warp == 0) {
        const int c = neh_warp(S, n, m);
        if (lane == 0) sh_cost = c;
        // visit order: the middle position first, then alternately right and left (IG.cpp:33-45)
        if (lane == 0) {
            const int start = n / 2;
            int ind = 0;
            for (int i = start; i < n; i++) { S.vo[ind] = i; ind += 2; }
            ind = 1;
            for (int i = start - 1; i >= 0; i--) { S.vo[ind] = i; ind += 2; }
        }
        __syncwarp();
        for (int i = lane; i < n; i += 32) { S.cur[i] = S.seq[i]; S.best[i] = S.seq[i]; }
    }
    __syncthreads();
    int cur_cost = sh_cost;
    int best_cost = cur_cost;
    long long sum = 0;
    for (int j = 0; j < n; j++) sum += S.tot[j];                // the jobs' total times, left by NEH
    const long long temp1000 = 20 * sum / ((long long)n * m);   // 1000 x 0.2 x mean / 10
    __syncthreads();
    int kmax = 1;
    while ((kmax + 1) * (kmax + 1) <= n) kmax++;   // integer square root
    int* Er = S.probe + warp * 2 * PBB_HEUR_REACH * PBB_HEUR_ROW;
    int* Qr = Er + PBB_HEUR_REACH * PBB_HEUR_ROW;
    unsigned long long rs = prm.seed + (unsigned long long)t;
    int perturb = prm.destruct;
    for (int it = 0; it < prm.iterations && n >= 3; it++) {
        if (warp == 0) {
            const int d = min(perturb, n - 1);
            for (int i = lane; i < n; i += 32) S.seq[i] = S.cur[i];
            __syncwarp();
            // destruction: d positions from a shuffled prefix of the visit order
            if (lane == 0) {
                const int r = rng_range(rs, d, n);
                for (int i = 0; i < r; i++) S.order[i] = S.vo[i];
                for (int i = 0; i < r - 1; i++) {
                    const int j = rng_range(rs, i, r - 1);
                    const int tmp = S.order[i]; S.order[i] = S.order[j]; S.order[j] = tmp;
                }
                // remove the chosen positions, highest first, keeping their jobs in draw order
                for (int i = 0; i < d; i++) removed[i] = S.seq[S.order[i]];
                for (int i = 0; i < n; i++) S.tot[i] = 0;
                for (int i = 0; i < d; i++) S.tot[S.order[i]] = 1;
                int w = 0;
                for (int i = 0; i < n; i++)
                    if (!S.tot[i]) S.seq[w++] = S.seq[i];
            }
            __syncwarp();
            // construction: each removed job at its best position
            int len = n - d, c = 0;
            for (int i = 0; i < d; i++) {
                const int x = removed[i];
                heads_tails(S.pt, S.mp, m, S.seq, len, S.E, S.Q);
                const unsigned long long key = best_insert(S.pt, S.mp, m, S.E, S.Q, x, len);
                insert_at(S.seq, len, (int)(key & 0xffffffffu), x);
                c = (int)(key >> 32);
                len++;
            }
            if (lane == 0) sh_cost = c;
        }
        __syncthreads();
        int cost = sh_cost;
        // local search: move the job at each visited position to the best
        // place within kmax of it, first improvement, until a pass finds none
        for (int pass = 0; pass < prm.ls_passes; pass++) {
            if (warp == 0) heads_tails(S.pt, S.mp, m, S.seq, n, S.E, S.Q);
            __syncthreads();
            int taken = -1;
            unsigned long long key = 0;
            for (int base = 0; base < n && taken < 0; base += warps) {
                const int j = base + warp;
                if (j < n) {
                    const unsigned long long b =
                        probe_move(S.pt, S.mp, n, m, S.seq, S.E, S.Q, S.vo[j], kmax, Er, Qr);
                    if (lane == 0) found[warp] = b;
                }
                __syncthreads();
                for (int w = 0; w < warps && base + w < n && taken < 0; w++) {
                    if ((int)(found[w] >> 32) < cost) {
                        taken = base + w;
                        key = found[w];
                    }
                }
                __syncthreads();
            }
            if (taken < 0) break;
            cost = (int)(key >> 32);
            if (warp == 0) {
                const int i = S.vo[taken];
                const int x = remove_at(S.seq, n, i);
                insert_at(S.seq, n - 1, (int)(key & 0xffffffffu), x);
            }
            __syncthreads();
        }
        // acceptance: one draw per round; not worse, or u / 2^32 < T / (T + delta)
        if (threadIdx.x == 0) {
            const long long delta = (long long)cost - cur_cost;
            const unsigned long long u = rng_next(rs) >> 32;
            sh_accept = (delta <= 0 || u < ((unsigned long long)temp1000 << 32) /
                                               (unsigned long long)(temp1000 + 1000 * delta)) ? 1 : 0;
        }
        __syncthreads();
        if (sh_accept) {
            if (warp == 0)
                for (int i = lane; i < n; i += 32) S.cur[i] = S.seq[i];
            cur_cost = cost;
            perturb = prm.destruct;
        } else {
            perturb = perturb + 1 > prm.destruct_max ? prm.destruct : perturb + 1;
        }
        if (cost < best_cost) {
            best_cost = cost;
            if (warp == 0)
                for (int i = lane; i < n; i += 32) S.best[i] = S.seq[i];
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) T.perm[i] = S.best[i];
    if (threadIdx.x == 0) {
        if (T.cost) *T.cost = best_cost;
        if (T.ub) *T.ub = best_cost;
    }
}

namespace pbbl {

cudaError_t launch_neh(const NehTask* tasks_d, int count, cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    cudaFuncSetAttribute(pbb_neh_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PBB_HEUR_SMEM);
    pbb_neh_kernel<<<count, 32, PBB_HEUR_SMEM, st>>>(tasks_d, count);
    return cudaGetLastError();
}

cudaError_t launch_ig(const NehTask* tasks_d, int count, const IgParams& prm, cudaStream_t st)
{
    if (count <= 0) return cudaSuccess;
    // eight warps whatever the count, although probes made for nothing then
    // cost other instances their turn: whole calls of 5 rounds with eight / two
    // warps, ms, 50x20 513 instances 3.1 / 4.3, 1024 5.4 / 6.6, 4096 19.0 / 19.7;
    // 20x10 1.3 / 1.4, 2.3 / 2.5, 8.8 / 8.7
    const int smem = PBB_HEUR_SMEM + PBB_IG_WARPS * PBB_IG_WARP_SMEM;
    cudaFuncSetAttribute(pbb_ig_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    pbb_ig_kernel<<<count, 32 * PBB_IG_WARPS, smem, st>>>(tasks_d, count, prm);
    return cudaGetLastError();
}

}  // namespace pbbl

namespace {

// Heuristic of `count` host instances on `device`; ig NULL = NEH alone.
int heur_batch(const pbb_instance* inst, int32_t count, int32_t device, const IgParams* ig, int32_t* perms,
               int32_t* costs)
{
    if (count < 0 || (count > 0 && (!inst || !perms || !costs))) return pbbt::fail(PBB_E_INVAL, "bad arguments");
    if (count == 0) return PBB_OK;
    size_t words = 0;
    for (int i = 0; i < count; i++) {
        const int n = inst[i].n_jobs, m = inst[i].n_machines;
        if (!inst[i].p || n < 1 || n > PBB_MAX_JOBS || m < 1 || m > PBB_MAX_MACHINES)
            return pbbt::fail(PBB_E_INVAL, "instance size out of range (1..64 jobs, 1..32 machines)");
        const int rc = pbbt::check_times(inst[i].p, n, m);
        if (rc) return rc;
        words += (size_t)n * m;
    }
    pbbh::DeviceGuard keep_callers_device;
    if (cudaSetDevice(device) != cudaSuccess) return pbbt::fail(PBB_E_CUDA, "cudaSetDevice failed");
    pbbh::Lease lease;
    if (pbbh::stream_take(&lease, device) != cudaSuccess) return pbbt::fail(PBB_E_CUDA, "stream creation failed");
    const cudaStream_t st = lease.st;
    unsigned char* d = nullptr;
    int rc = PBB_OK;
    do {
        const size_t out_words = (size_t)count * (PBB_MAX_JOBS + 1);
        pbbh::Carver C;
        const size_t o_tasks = C.take(sizeof(NehTask) * count), o_p = C.take(sizeof(int) * words);
        const size_t filled = C.bytes;
        const size_t o_out = C.take(sizeof(int) * out_words);
        if (pbbh::mem_alloc((void**)&d, C.bytes, lease) != cudaSuccess) {
            rc = pbbt::fail(PBB_E_NOMEM, "device allocation failed");
            break;
        }
        std::vector<unsigned char> host(filled);
        NehTask* tasks = reinterpret_cast<NehTask*>(host.data() + o_tasks);
        int* times = reinterpret_cast<int*>(host.data() + o_p);
        int* out = reinterpret_cast<int*>(d + o_out);
        size_t off = 0;
        for (int i = 0; i < count; i++) {
            const int n = inst[i].n_jobs, m = inst[i].n_machines;
            memcpy(times + off, inst[i].p, sizeof(int) * n * m);
            tasks[i].p = reinterpret_cast<int*>(d + o_p) + off;
            tasks[i].n = n;
            tasks[i].m = m;
            tasks[i].perm = out + (size_t)i * (PBB_MAX_JOBS + 1);
            tasks[i].cost = out + (size_t)i * (PBB_MAX_JOBS + 1) + PBB_MAX_JOBS;
            tasks[i].ub = nullptr;
            off += (size_t)n * m;
        }
        const NehTask* tasks_d = reinterpret_cast<const NehTask*>(d + o_tasks);
        cudaError_t ce = cudaMemcpyAsync(d, host.data(), filled, cudaMemcpyHostToDevice, st);
        if (!ce) ce = ig ? pbbl::launch_ig(tasks_d, count, *ig, st) : pbbl::launch_neh(tasks_d, count, st);
        std::vector<int> res(out_words);
        if (!ce) ce = cudaMemcpyAsync(res.data(), out, sizeof(int) * out_words, cudaMemcpyDeviceToHost, st);
        if (!ce) ce = cudaStreamSynchronize(st);
        if (ce) {
            rc = pbbt::fail(PBB_E_CUDA, cudaGetErrorString(ce));
            break;
        }
        for (int i = 0; i < count; i++) {
            const int* row = res.data() + (size_t)i * (PBB_MAX_JOBS + 1);
            const int n = inst[i].n_jobs;
            int32_t* to = perms + (size_t)i * PBB_MAX_JOBS;
            memcpy(to, row, sizeof(int) * n);
            memset(to + n, 0, sizeof(int) * (PBB_MAX_JOBS - n));
            costs[i] = row[PBB_MAX_JOBS];
        }
    } while (0);
    cudaStreamSynchronize(st);
    pbbh::mem_free(d, lease);
    pbbh::stream_give(lease);
    return rc;
}

}  // namespace

extern "C" int pbb_neh_batch(const pbb_instance* inst, int32_t count, int32_t device, int32_t* perms,
                             int32_t* costs)
{
    return heur_batch(inst, count, device, nullptr, perms, costs);
}

extern "C" int pbb_ig_batch(const pbb_instance* inst, int32_t count, int32_t device, int32_t iterations,
                            uint64_t seed, int32_t* perms, int32_t* costs)
{
    if (iterations < 0 || iterations > 100000) return pbbt::fail(PBB_E_INVAL, "iterations must be in [0, 100000]");
    IgParams prm;
    prm.iterations = iterations;
    prm.destruct = 2;          // IG::destructStrength (heuristic/src/IG.cpp:22)
    prm.destruct_max = 5;      // perturbation cap (IG.cpp:393-396)
    prm.ls_passes = 64;
    prm.seed = seed;
    return heur_batch(inst, count, device, &prm, perms, costs);
}
