// Device heuristics (pbb_heur.cu): NEH, one warp per instance, and iterated
// greedy, eight.
#pragma once
#include <cuda_runtime.h>
#include "pbb_types.h"

// One instance for the heuristic kernels (device pointers).
struct NehTask {
    const int* p;   // [m][n] processing times
    int n, m;
    int* perm;      // [n] result permutation
    int* cost;      // result makespan (may be NULL)
    int* ub;        // also written here when not NULL (an explorer group's initial bound)
};

// Iterated greedy settings (pbb_ig_batch); the same stream of decisions on
// host and device for the same seed.
struct IgParams {
    int iterations;          // destruction / construction / local-search rounds
    int destruct;            // jobs removed per round at first (grows to destruct_max on failures)
    int destruct_max;
    int ls_passes;           // insertion local-search passes per round at most
    unsigned long long seed;
};

// Row stride of the heads and tails kept by position: with 34 ints neither the
// wavefront's diagonal stores nor the reads of one machine at many positions
// meet on a bank more than twice.
#define PBB_HEUR_ROW 34
#define PBB_HEUR_REACH 8          // local-search moves reach at most sqrt(64) places
#define PBB_IG_WARPS 8            // warps of an iterated-greedy block
// shared memory of one heuristic block: p, heads, tails, and per-job arrays;
// and of each local-search warp: the rows its probe computes anew
#define PBB_HEUR_SMEM (int)(sizeof(int) * (PBB_MAX_N * 36 + (2 * PBB_MAX_N + 1) * PBB_HEUR_ROW + 6 * PBB_MAX_N))
#define PBB_IG_WARP_SMEM (int)(sizeof(int) * 2 * PBB_HEUR_REACH * PBB_HEUR_ROW)

namespace pbbl {
cudaError_t launch_neh(const NehTask* tasks_d, int count, cudaStream_t st);
cudaError_t launch_ig(const NehTask* tasks_d, int count, const IgParams& prm, cudaStream_t st);
}
