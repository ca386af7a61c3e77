"""Shared-memory layout of a CTA: the padded rows of the processing times and
the work-sharing block cost no instance a warp, and no pool its block shape,
that unpadded tables have room for."""
import ctypes
import os
import subprocess

import pytest

from oracle import Oracle
import pbbperm_b200 as pb
from pbbperm_b200.instances import synthetic_instance

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMEM = 232448          # shared memory a block may ask for (227 KiB)
SHIM = r"""
#include "pbb_types.h"
extern "C" int plan_total(int n, int m, int Ppad, int warps, int scratch)
{
    return pbb_smem_plan(n, m, Ppad, warps, scratch).total;
}
extern "C" int plan_stride(int n, int m, int Ppad, int warps, int scratch)
{
    return pbb_smem_plan(n, m, Ppad, warps, scratch).je_stride;
}
// the first instance of at most n x m whose plan a launch sized for n x m does
// not hold, 0 when there is none
extern "C" int first_too_large(int n, int m, int warps, int scratch)
{
    const int room = pbb_smem_plan(n, m, (m * (m - 1) / 2 + 31) / 32 * 32, warps, scratch).total;
    for (int i = 1; i <= n; i++)
        for (int k = 1; k <= m; k++)
            for (int Ppad = (k * (k - 1) / 2 + 31) / 32 * 32; Ppad >= 0; Ppad -= 32)
                if (pbb_smem_plan(i, k, Ppad, warps, scratch, room).total > room) return i * 100 + k;
    return 0;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SHIM)
    so = str(d / "plan.so")
    subprocess.check_call(["g++", "-w", "-shared", "-fPIC", "-O1", "-std=c++17", "-include", "cuda_runtime.h",
                           "-I", "/usr/local/cuda/include", "-I", os.path.join(ROOT, "pbbperm_b200", "csrc"),
                           "-o", so, str(d / "plan.cpp")])
    return ctypes.CDLL(so)


def up(x, a):
    return (x + a - 1) // a * a


def tight_total(n, m, ppad, warps, masks):
    """Tables with rows of exactly m times, and the general build's scratch."""
    tables = n * ppad * 8 + up(4 * m * n, 16) + 2 * up(ppad, 16) + 2 * up(4 * m, 16) + up(n * ppad, 16)
    warp = up((8 * ppad if masks else 0) + (2 * n + 7 * 32) * 4 + 4 * n * m + 3 * n, 16)
    return tables + warps * warp


def test_what_fits_unpadded_fits(shim):
    for n in range(1, 65):
        for m in range(2, 33):
            for pairs in {m * (m - 1) // 2, m - 1}:
                ppad = up(pairs, 32)
                for scratch in (0, 1):
                    for warps in range(1, 21):
                        if tight_total(n, m, ppad, warps, scratch) > SMEM:
                            break
                        assert shim.plan_total(n, m, ppad, warps, scratch) <= SMEM, (n, m, pairs, scratch, warps)


def test_rows_are_padded_wherever_that_costs_no_cta(shim):
    """Tight rows are for the tables that need them: the rows of 20-machine
    instances stay a multiple of 32 entries."""
    for n in range(2, 51):
        for scratch in (0, 1):
            assert shim.plan_stride(n, 20, 192, 20, scratch) == 192, (n, scratch)
    assert shim.plan_stride(43, 30, 448, 8, 0) == 435


@pytest.mark.parametrize("warps", [1, 4, 8, 16, 20])
def test_a_launch_holds_every_smaller_instance(shim, warps):
    """A pool sizes its launches for its largest instance; a smaller one is never
    larger, whichever rows either has."""
    for n, m in [(12, 10), (22, 20), (43, 30), (53, 27), (43, 32), (52, 29), (61, 26), (60, 21), (41, 25), (61, 17),
                 (22, 29), (59, 16), (64, 20), (64, 5)]:
        for scratch in (0, 1, 2, 3):
            assert shim.first_too_large(n, m, warps, scratch) == 0, (n, m, scratch)


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,ub", [(43, 30, 3879), (53, 27, 4170)])
def test_pools_at_the_shared_memory_limit(n, m, ub):
    """The largest pools eight warps a CTA have room for."""
    p = synthetic_instance(1, n, m)
    want = Oracle(p).solve(ub, bound_mode=2)
    assert want["complete"] and not want["found"] and want["decomposed"] > 500
    with pb.Pool(pb.PoolConfig(max_jobs=n, max_machines=m, max_resident=2)) as pool:
        for t in range(3):
            pool.submit(p, tag=t, ub=ub, config=pb.Config(boundingMode=2))
        got = {}
        for _ in range(1000):
            pool.step()
            got.update((r["tag"], r) for r in pool.poll())
            if len(got) == 3:
                break
    assert sorted(got) == [0, 1, 2]
    for r in got.values():
        assert r["status"] == pb.PBB_OK and r["complete"]
        for k in ("decomposed", "johnson_bounds", "simple_bounds", "leaves"):
            assert r[k] == want[k], (k, r[k], want[k])
