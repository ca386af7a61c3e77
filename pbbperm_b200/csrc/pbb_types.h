// Shared host/device definitions of the IVM flow-shop engine.
#pragma once
#include <stdint.h>

#define PBB_MAX_N 64          // jobs per instance (int8 IVM cells, two 32-bit mask words)
#define PBB_MAX_M 32          // machines per instance (one machine per lane in recurrences)
#define PBB_WARPS_MAX 20      // explorer warps per CTA (96 registers a thread)
// Warps of an explorer CTA at most: 20 at 96 registers a thread, or 32 at 64
// in the wide builds of the variants with kept pair bounds (5 and 6, of 3 and
// 4), whose scratch leaves the room.
#define PBB_WIDE_WARPS 32
#define PBB_EXPLORE_WARPS(var) ((var) == 5 || (var) == 6 ? PBB_WIDE_WARPS : PBB_WARPS_MAX)
// What an explorer variant bounds with (pbb_launch.h): kept pair bounds, with
// the search's settings at run time, or every child's Johnson value; and
// whether it records sampled nodes
#define PBB_VAR_PAIRS(var) (((var) >= 3 && (var) <= 6) || (var) == 8 || (var) == 9)
#define PBB_VAR_GEN(var) ((var) == 4 || (var) == 6 || (var) == 9)
#define PBB_VAR_ALL(var) ((var) == 7 || (var) == 10)
#define PBB_VAR_SAMPLE(var) ((var) == 2 || (var) >= 8)
// The wide builds gain 14 to 20 % where a search is long and its instance has
// many machine pairs, and lose 6 to 10 % where either is missing: a short
// search is bound by the time one node takes and by how fast work spreads, and
// with few pairs there is little to overlap for the spilled registers.  The
// size of the tree is not known beforehand; the instance's size is what there is
// to go by.  Explorer ms with 20 and with 32 warps:
//   used from here on: 20x20 (13 M nodes) 38.9 and 32.0, 18x20 (19 M) 55.6 and
//   44.7, 33x15 (35 M) 96.8 and 79.0, 30x20 (54 M) 131 and 106, 40x20 (60 M) 190
//   and 164, 50x20 (56 M) 194 and 167; but 18x20 (0.9 M) 3.3 and 3.6, (0.6 M) 2.4
//   and 2.6, 25x20 (2.6 M) 7.3 and 7.9, 40x10 (0.3 M) 2.1 and 2.2;
//   not used: 16x20 (1.9 M) 6.1 and 6.5, 30x10 (10 M) 20.8 and 22.7, 24x10
//   (0.5 M) 1.6 and 1.8, 14x20 (0.2 M) 1.16 and 1.29, 12x10 0.21 and 0.23.
#define PBB_WIDE_FROM 320             // jobs x machines above which they are used
// warps of a bound kernel's CTA at most, by the 32-job words of a row: two
// words leave shared memory for fewer, and want more registers
#define PBB_BOUND_WARPS(nw) ((nw) == 1 ? 16 : 12)
#define PBB_CORE_WARPS PBB_WARPS_MAX   // default of DevSearch::core_warps: all but 12 in a wide build
#define PBB_SPLIT_DEPTH 10    // default of DevSearch::split_depth
#define PBB_SHARE_AFTER 64    // default of DevSearch::share_after
#define PBB_SPLIT_NARROW 4    // default of DevSearch::split_narrow
#define PBB_FLUSH_NODES (1u << 10)     // nodes after which a warp adds its counters to the group's

// IVM life cycle (per explorer, in global memory)
#define IVM_IDLE 0            // no interval
#define IVM_ACTIVE 2          // holds a non-empty interval

// status bits written by kernels (never traps)
#define PBB_ST_BADINPUT 1u    // a node or instance the kernel rejected

// Packed Johnson entry for (pair i, Johnson position t):
//   bits 0..15 p[m0][job], 16..31 p[m1][job], 32..39 job id, 40..63 lag[i][job]
// (the two processing times share the low word, so the scans unpack them with
// one mask and one shift)
#define JE_PACK(job, a, b, lag) ((unsigned long long)(a) | ((unsigned long long)(b) << 16) | \
                                 ((unsigned long long)(job) << 32) | ((unsigned long long)(lag) << 40))
#define JE_A(e) ((int)((unsigned)(e) & 0xFFFFu))
#define JE_B(e) ((int)((unsigned)(e) >> 16))
#define JE_JOB(e) ((int)(((e) >> 32) & 0xFFull))
#define JE_C(e) ((int)((e) >> 40))

// One flow-shop instance as the kernels see it (device pointers).
struct DevInstance {
    int n, m;
    int P;        // machine pairs used by the Johnson bound
    int Ppad;     // P rounded up to 32
    const int* p;                    // [m][n]
    const unsigned long long* je;    // [n][Ppad]
    const unsigned char* posj;       // [n][Ppad] Johnson position of each job per pair (may be NULL)
    const unsigned char* pm0;        // [Ppad]
    const unsigned char* pm1;        // [Ppad]
    const int* min_arr;              // [m]
    const int* min_dep;              // [m]
};

// Search settings shared by a group of explorers.
struct DevSearch {
    int bound_mode;    // 0 weak, 1 strong, 2 weak then strong
    int branch_mode;   // -3,-2,-1 fixed; 1 MaxSum, 2 MinBranch, 3 MinMin
    int find_all;
    int sort_nodes;    // [bb] sortedDFS: 0 reverse the row on a side change, 1 sort it by cost,
                       //      2 and 4 by (cost, priority), 3 by priority
    int sort_crit;     // [bb] sortingCriterion (sortedDFS >= 2): 1 cost, 2 cost minus the other side's, 3 idle time
    int early_stop;    // [bb] earlyStopJohnson: a child's Johnson scan may stop once it exceeds the incumbent
    int core_warps;    // warps per CTA that ask for work whatever the search's width (1..warps per CTA)
    int split_depth;   // work is not split at levels deeper than n - split_depth
    int split_narrow;  // the same limit while most warps of the CTA, or most CTAs, wait for work
    int share_after;   // an explorer gives work away only after decomposing this many nodes since it
                       // got its interval or last gave part of it away, fewer the more warps wait
                       // (0 = at every step)
};

// Per-group control block (device memory).
// The incumbent and the count of waiting CTAs are read together by every
// working warp; the active count, which every start and end of an interval
// updates, sits on a line of its own.
struct GroupCtl {
    alignas(128) unsigned long long best_key;   // (cost << 32) | ivm id of the slot holding the permutation
    int asking;                                 // CTAs asking other CTAs for work
    alignas(128) int active;                    // explorers holding work
    alignas(128) int found;                     // leaves that improved (or matched, with findAll) the bound
    unsigned int status;                        // PBB_ST_* bits
    unsigned long long decomposed, johnson_bounds, simple_bounds, leaves, root_simple;
    unsigned long long steals;                  // intervals handed over
    // work of the Johnson sweeps: nodes swept, free jobs summed over them,
    // children evaluated by them (roofline accounting)
    unsigned long long jsweeps, jfree, jchild;
    // children bounded by direct scans, and free jobs summed over the machine
    // pairs scanned for them (kept pair bounds: children compared, positions
    // of the pairs scanned)
    unsigned long long jdirect, jdirect_free;
};

// Explorer storage of a group (device memory, structure of arrays).
struct DevIvms {
    int count;             // explorers in the group
    int npad;              // row stride (32 for up to 32 jobs, else 64)
    int levels;            // levels kept of each explorer (at least the jobs)
    signed char* mat;      // [count][levels][npad]
    signed char* pos;      // [count][npad]
    signed char* end;      // [count][npad]
    signed char* dir;      // [count][npad]
    signed char* pj;       // [count][npad] job fixed at each level of the current path
    int* line;             // [count]
    int* state;            // [count]
    int* bestcost;         // [count]
    signed char* bestperm; // [count][npad]
    unsigned int* ask;     // [(count + 31) / 32] bit c: CTA c of the group asks for work
    int* askid;            // [count] explorer that asking CTA c offers for it
    int* path;             // [count][levels][3][32] heads / tails / free loads of the path nodes
};

#define PBB_PATH_INTS 96   // ints per path level: heads, tails, free loads, 32 machines each

// Opt-in record of nodes the explorer bounded, as it bounded them (LB parity
// of the explorer's own bound code).  A node is recorded when a hash of
// (explorer id, the warp's decomposed count) has its low bits clear under
// rate_mask, until `cap` records are taken; recording never waits.
// Record layout (ints): PBB_SAMPLE_HDR header
//   [0] explorer id  [1] line  [2] limit1  [3] limit2  [4] side chosen
//   [5] incumbent at bounding  [6] free jobs k  [7] 0
// then five arrays of n: schedule (front jobs, free jobs, back jobs as the
// reference's node->schedule), weak LB front / back and Johnson LB front /
// back by job id (0 = not evaluated).
#define PBB_SAMPLE_HDR 8
struct SampleBuf {
    unsigned count;        // records claimed (may exceed cap; only cap are written)
    unsigned cap;
    unsigned rate_mask;
    int stride;            // ints per record: PBB_SAMPLE_HDR + 5 n
    int* rec;
};

struct DevGroup {
    DevInstance inst;
    DevSearch search;
    DevIvms ivm;
    GroupCtl* ctl;
    int first_cta;         // CTAs [first_cta, first_cta + ctas) work on this group
    int ctas;
    SampleBuf* sample;     // NULL unless node sampling is armed
};

// Optional outputs of the bound kernel (NULL = not wanted): per node and job,
// the children's idle-time priorities, and per node the Johnson bound's idle
// time of the fixed jobs.
struct BoundExtra {
    int* prio_begin = nullptr;   // [count][n]
    int* prio_end = nullptr;     // [count][n]
    int* strong_idle = nullptr;  // [count]
};

// Work sharing inside one CTA (shared memory): a warp without work sets its
// bit in `hungry` after writing the explorer it offers; a working warp that
// splits its interval clears a bit, fills that explorer and posts its id in
// the waiting warp's mail.
struct CtaShare {
    unsigned hungry;       // warps waiting for work
    int working;           // warps holding work
    int asker;             // 1 + the warp that asks other CTAs for this one (0: none)
    int stop;              // the group's search has ended
    int active;            // last value read of the group's active count
    int best;              // last value read of the incumbent
    int asking;            // last value read of the group's waiting CTAs
    unsigned poll_ns;      // when the group's active count was last read (low word of the timer)
    // int offer[warps], mail[warps] follow
};

// Dynamic shared memory layout of one CTA (host and device agree).
struct SmemPlan {
    int je_off, p_off, pre_off, pm_off, marr_off, mdep_off, posj_off, share_off, warp_off, warp_bytes, total;
    int je_stride;         // entries between rows of the Johnson table
    int posj_stride;       // bytes between rows of the position table
    int fmask;             // PBB_SCRATCH_*
};

// Per-warp scratch of the kernels
#define PBB_SCRATCH_PLAIN 0   // no free-position masks
#define PBB_SCRATCH_MASKS 1   // with the masks of the explorer the warp holds
#define PBB_SCRATCH_PAIRS 2   // kept pair bounds (bounding mode 2), no per-child tables
#define PBB_SCRATCH_ALL 3     // Johnson values of every child of both sides (bound kernel, bounding mode 1)

__host__ __device__ inline int pbb_align(int x, int a) { return (x + a - 1) / a * a; }

// Row stride (ints) of the processing times kept job by job in shared memory:
// machines rounded up to an odd number of 16-byte words, so that the lanes of
// a warp read four machines of 32 different jobs without bank conflicts.
__host__ __device__ inline int pbb_machine_pad(int m) { return ((m + 3) / 4 | 1) * 4; }

// per-warp scratch: ints Fb Bb RB FR frontZ backZ rem [32 each], then
// [fmask: u64 fmask[Ppad]] ints lbF[n] lbB[n]; shorts dF[n*m] dB[n*m]; bytes
// fjob[n] bjob[n] row[n].  PBB_SCRATCH_PAIRS has, in place of fmask lbF lbB dF
// dB: ints the child's vectors [128], two pair-bound buffers [Ppad each];
// PBB_SCRATCH_ALL: ints a warp pass's pairs [128], their values by position
// [n][33]; shorts dF dB [m][32 or 64 children each]
__host__ __device__ inline int pbb_warp_bytes(int n, int m, int Ppad, int fmask)
{
    if (fmask == PBB_SCRATCH_PAIRS) return pbb_align((7 * 32 + 128 + 2 * Ppad) * 4 + 3 * n, 16);
    if (fmask == PBB_SCRATCH_ALL)
        return pbb_align((7 * 32 + 128 + n * 33) * 4 + 2 * m * (n <= 32 ? 32 : 64) * 2 + 3 * n, 16);
    return pbb_align((fmask ? Ppad * 8 : 0) + (2 * n + 7 * 32) * 4 + 2 * n * m * 2 + 3 * n, 16);
}

// PBB_SCRATCH_PAIRS keeps no position table, but the prefix sums of the
// processing times, and an odd row stride of the Johnson entries, so that a
// warp can read one pair's column as well as 32 pairs' rows.
// CTAs of `warps` warps at 96 registers a thread that an SM holds (228 KiB of
// shared memory, 1 KiB of it reserved for each)
__host__ __device__ inline int pbb_sm_ctas(int total, int warps)
{
    const int regs = warps < 21 ? 21 / warps : 1, smem = 233472 / (total + 1024);
    return smem < regs ? smem : regs;
}

// Rows of the Johnson table hold Ppad entries, so that lanes at different
// positions of their pairs' orders meet no bank twice; without what is past the
// last pair (whatever the Johnson mode, there are no more than machine pairs)
// they take less memory, and bounding mode 1 at 50x20 runs 7 % slower.  Tight rows
// are for tables that need it: on the host (room < 0), where the padded rows of
// the processing times and the work-sharing block would cost the SM a CTA; in a
// kernel, whose launch has `room` bytes, where the padded rows do not fit them.
__host__ __device__ inline SmemPlan pbb_smem_plan(int n, int m, int Ppad, int warps, int fmask = 0, int room = -1)
{
    const bool pairs = fmask == PBB_SCRATCH_PAIRS, general = !pairs && fmask != PBB_SCRATCH_ALL;
    const int times = n * pbb_machine_pad(m) * 4, share = pbb_align((int)sizeof(CtaShare) + 8 * warps, 16);
    const int last = m * (m - 1) / 2, tight = last < Ppad ? last : Ppad;
    SmemPlan s;
    s.je_stride = pairs ? Ppad + 1 : Ppad;
    for (int pass = 0; pass < 2; pass++) {
        int off = 0;
        s.je_off = off;   off += pbb_align(n * s.je_stride * 8, 16);
        s.p_off = off;    off += times;
        s.pre_off = off;  off += pairs ? times : 0;
        s.pm_off = off;   off += pbb_align(Ppad * 2, 16);
        s.marr_off = off; off += pbb_align(m * 4, 16);
        s.mdep_off = off; off += pbb_align(m * 4, 16);
        // an odd number of words between the rows of the position table lets the
        // lanes read one pair's positions of 32 jobs without bank conflicts; the
        // general builds read one job's row, and use one stride for both tables
        s.posj_stride = fmask == PBB_SCRATCH_ALL ? Ppad + 4 : s.je_stride;
        s.posj_off = off; off += pairs ? 0 : pbb_align(n * s.posj_stride, 16);
        s.share_off = off; off += share;
        s.warp_off = off;
        s.fmask = fmask;
        s.warp_bytes = pbb_warp_bytes(n, m, Ppad, fmask);
        off += s.warp_bytes * warps;
        s.total = off;
        const int grown = times - pbb_align(4 * m * n, 16) + share;
        if (!general || (room < 0 ? pbb_sm_ctas(off, warps) >= pbb_sm_ctas(off - grown, warps) : off <= room)) break;
        s.je_stride = tight;
    }
    return s;
}
