// Host-callable launch wrappers of the engine kernels (pbb_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include "pbb_types.h"

namespace pbbl {
// The explorer variant with kept pair bounds for a search's settings, 0 when
// there is none: mode 2 with a rule that bounds the side it chooses (-2 and -3
// choose the back side without its weak bound, so Johnson values stand alone).
inline int pairs_variant(int bound_mode, int branch_mode, int find_all, int sort_nodes)
{
    if (bound_mode != 2 || branch_mode < -1) return 0;
    return branch_mode == 3 && !find_all && !sort_nodes ? 3 : 4;
}

// dynamic shared memory of a CTA; fmask: the per-warp scratch (PBB_SCRATCH_*)
int smem_bytes(int n, int m, int Ppad, int warps, int fmask = 0);
cudaError_t launch_reset(const DevGroup* groups, int ngroups, const int* ub, cudaStream_t st);
// reset must run first; interval b = g * per_group + j starts explorer j of
// group g, or explorer ids[b] when ids is given (distinct, < the explorer count)
cudaError_t launch_root(int nw, const DevGroup* groups, int ngroups, const int* roots, const int* ivals,
                        int root_stride, int smem, cudaStream_t st, int per_group = 1, const int* ids = nullptr);
cudaError_t launch_lower_ub(const DevGroup* groups, int g, int ub, cudaStream_t st);
// variant: 0 = no row sort, no early Johnson exit, no sampling; 1 = each
// group's sortedDFS / earlyStopJohnson settings; 2 = as 1 and record sampled
// nodes (groups' SampleBuf); 3 to 6 = kept pair bounds (pairs_variant; 5 and 6
// for up to PBB_WIDE_WARPS a CTA), launched
// with the PBB_SCRATCH_PAIRS shared memory and with pair_stack, pair_stride
// ints for each warp of the grid (at least jobs x padded machine pairs).
// 7 = every child's Johnson value (mode 1, up to 32 jobs), launched with the
// PBB_SCRATCH_ALL shared memory.  8, 9 and 10 = as 3, 4 and 7 and record sampled
// nodes.
// eager = 0: a short window, which splits work only as often as share_after
// says, however many warps wait
cudaError_t launch_explore(int nw, const DevGroup* groups, const int* ngroups_d, int ctas, int warps_per_cta, int smem,
                           unsigned long long budget_ns, int max_rounds, int select_budget, cudaStream_t st,
                           int variant = 0, int eager = 1, int* pair_stack = nullptr, int pair_stride = 0);
// resident CTAs of the variants a pool launches (0, 3, 4)
int explore_ctas_per_sm(int nw, int warps_per_cta, int smem, int variant = 0);
// The launch of a batch of `count` nodes: kernel and block shape that fit
// `optin` bytes of shared memory (warps 0: none does)
struct BoundShape {
    bool all = false;      // pbb_bound_all_kernel
    int warps = 0, ctas = 1, smem = 0;
};
BoundShape bound_shape(int n, int m, int Ppad, int count, int sms, int optin);
cudaError_t launch_bound_all(int nw, const DevInstance& I, int count, const int* sched, const int* l1, const int* l2,
                             int* wb, int* we, int* sb, int* se, int* nweak, int* nstrong, unsigned int* status,
                             const BoundShape& b, cudaStream_t st, BoundExtra extra = BoundExtra());
// method (diagnostic): 0 sweeps over all positions, 1 direct scans, 2 sweeps over the free positions
cudaError_t launch_bound(int nw, const DevInstance& I, int count, const int* sched, const int* l1, const int* l2,
                         int* wb, int* we, int* sb, int* se, int* nweak, int* nstrong, unsigned int* status, int ctas,
                         int warps_per_cta, int smem, cudaStream_t st, int method = 0, BoundExtra extra = BoundExtra());
}  // namespace pbbl
