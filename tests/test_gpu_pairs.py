"""Bounding mode 2 by kept pair bounds: the children pruned are those of the
full Johnson bound, so every counter equals the oracle's -- over one and two
words of jobs and their edges, one to 496 machine pairs, machines at and
around the 16-byte steps of the one-machine bound, every JohnsonMode, and the
rules and options that take this path or the general one (-2)."""
import pytest

from oracle import Oracle
import pbbperm_b200 as pb
from pbbperm_b200.instances import synthetic_instance

pytestmark = pytest.mark.gpu

KEYS = ("decomposed", "johnson_bounds", "simple_bounds", "leaves")

# jobs, machines, JohnsonMode, seed, a value below every schedule
CASES = [(12, 10, 1, 3, 1171), (12, 10, 2, 3, 1171), (16, 12, 0, 2, 1525), (32, 10, 0, 3, 2141), (33, 10, 0, 3, 2093),
         (14, 20, 0, 1, 1915), (18, 32, 0, 5, 2741), (40, 10, 0, 4, 2439), (64, 10, 0, 4, 3773), (50, 20, 0, 3, 3624)]
OPTIONS = [dict(), dict(adaptiveBranchingMode=1), dict(adaptiveBranchingMode=2, findAll=True),
           dict(adaptiveBranchingMode=-1, sortedDFS=2, sortingCriterion=2), dict(earlyStopJohnson=True, sortedDFS=1),
           dict(adaptiveBranchingMode=-2)]


@pytest.mark.parametrize("n,m,jmode,seed,ub", CASES)
@pytest.mark.parametrize("opt", OPTIONS, ids=[str(i) for i in range(len(OPTIONS))])
def test_counts_equal_the_oracle(n, m, jmode, seed, ub, opt):
    rule = opt.get("adaptiveBranchingMode", 3)
    if rule == -2 and n > 16:
        pytest.skip("back branching alone grows trees too large for the oracle")
    if rule == -1 and n not in (12, 16, 64):
        pytest.skip("front branching alone grows trees too large for the oracle")
    p = synthetic_instance(seed, n, m)
    ub -= 1 if opt.get("findAll") else 0
    want = Oracle(p, jmode).solve(ub, bound_mode=2, branch_mode=rule, find_all=opt.get("findAll", False),
                                  sorted_dfs=opt.get("sortedDFS", 0),
                                  sorting_criterion=opt.get("sortingCriterion", 1), node_limit=60000)
    if not want["complete"]:
        pytest.skip("the tree is too large for the oracle")
    assert not want["found"]
    cfg = pb.Config(boundingMode=2, JohnsonMode=jmode, nbIVMs=4096, **opt)
    with pb.Engine(p, cfg) as e:
        got = e.solve(ub=ub)
    assert got["complete"] and not got["found"]
    for k in KEYS:
        assert got[k] == want[k], (k, got[k], want[k])


@pytest.mark.parametrize("n,m", [(2, 2), (3, 2), (4, 3), (5, 4), (6, 5), (7, 32)])
def test_smallest_rows_from_no_bound(n, m):
    """One explorer from +inf visits the nodes in the oracle's order, so the
    counters agree although the incumbent improves on the way."""
    p = synthetic_instance(n + m, n, m)
    want = Oracle(p).solve(2**31 - 1, bound_mode=2)
    with pb.Engine(p, pb.Config(boundingMode=2, nbIVMs=1)) as e:
        got = e.solve()
    assert got["complete"] and got["cost"] == want["best"]
    for k in KEYS:
        assert got[k] == want[k], (k, got[k], want[k])


@pytest.mark.parametrize("n,m,seed,ub", [(12, 10, 3, 1171), (13, 10, 3, 1277), (9, 20, 2, 1400), (32, 10, 3, 2110),
                                         (33, 10, 3, 2070), (14, 32, 1, 2300)])
@pytest.mark.parametrize("opt", [dict(), dict(adaptiveBranchingMode=2, sortedDFS=1), dict(adaptiveBranchingMode=1),
                                 dict(adaptiveBranchingMode=-1, findAll=True)], ids=["0", "1", "2", "3"])
def test_mode_1_counts_equal_the_oracle(n, m, seed, ub, opt):
    """Bounding mode 1, rows of one word (values by position) and of two: small
    trees, many of a handful of nodes; trees of size are below."""
    p = synthetic_instance(seed, n, m)
    want = Oracle(p).solve(ub, bound_mode=1, branch_mode=opt.get("adaptiveBranchingMode", 3),
                           find_all=opt.get("findAll", False), sorted_dfs=opt.get("sortedDFS", 0), node_limit=20000)
    if not want["complete"] or want["found"]:
        pytest.skip("not a small proof")
    with pb.Engine(p, pb.Config(boundingMode=1, nbIVMs=4096, **opt)) as e:
        got = e.solve(ub=ub)
    assert got["complete"] and not got["found"]
    for k in KEYS:
        assert got[k] == want[k], (k, got[k], want[k])


# jobs, machines, JohnsonMode, seed, a value below every schedule, the options,
# and the oracle's nodes: trees that cannot pass without being searched
TREES = [
    # the front rule alone computes the one-machine bounds of one side
    (20, 10, 0, 1, 1528, dict(boundingMode=2, adaptiveBranchingMode=-1), 2141),
    (16, 12, 0, 2, 1466, dict(boundingMode=2, adaptiveBranchingMode=-1), 8182),
    (14, 20, 0, 1, 1886, dict(boundingMode=2, adaptiveBranchingMode=-1, sortedDFS=2, sortingCriterion=2), 2923),
    # findAll keeps children at the bound
    (16, 12, 0, 2, 1498, dict(boundingMode=2, adaptiveBranchingMode=2, findAll=True), 2702),
    (16, 12, 2, 2, 1498, dict(boundingMode=2, adaptiveBranchingMode=2, findAll=True), 5013),
    (14, 32, 1, 1, 2521, dict(boundingMode=2, adaptiveBranchingMode=2, findAll=True), 5883),
    # mode 1, 17 to 32 free jobs a row
    (20, 20, 0, 1, 2254, dict(boundingMode=1, adaptiveBranchingMode=1), 2653),
    (20, 20, 0, 1, 2254, dict(boundingMode=1, adaptiveBranchingMode=2, findAll=True), 2351),
    (24, 20, 0, 1, 2272, dict(boundingMode=1, adaptiveBranchingMode=-1, findAll=True), 7743),
    (32, 20, 0, 2, 2994, dict(boundingMode=1, adaptiveBranchingMode=-1, findAll=True), 4669),
    (14, 32, 0, 1, 2576, dict(boundingMode=1, adaptiveBranchingMode=-1, findAll=True), 2537),
]


@pytest.mark.parametrize("n,m,jmode,seed,ub,opt,nodes", TREES)
def test_counts_of_whole_trees(n, m, jmode, seed, ub, opt, nodes):
    p = synthetic_instance(seed, n, m)
    want = Oracle(p, jmode).solve(ub, bound_mode=opt["boundingMode"], branch_mode=opt.get("adaptiveBranchingMode", 3),
                                  find_all=opt.get("findAll", False), sorted_dfs=opt.get("sortedDFS", 0),
                                  sorting_criterion=opt.get("sortingCriterion", 1))
    assert want["decomposed"] == nodes and not want["found"]
    with pb.Engine(p, pb.Config(JohnsonMode=jmode, nbIVMs=4096, **opt)) as e:
        got = e.solve(ub=ub)
    assert got["complete"] and not got["found"]
    for k in KEYS:
        assert got[k] == want[k], (k, got[k], want[k])


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("opt", [dict(), dict(adaptiveBranchingMode=2), dict(adaptiveBranchingMode=-1)],
                         ids=["3", "2", "-1"])
def test_find_all_counts_every_optimum(mode, opt):
    """findAll from the optimum: the incumbent cannot improve, so the counters
    do not depend on the order, and every optimal leaf is reached."""
    p = synthetic_instance(3, 12, 10)
    rule = opt.get("adaptiveBranchingMode", 3)
    want = Oracle(p).solve(1171, bound_mode=mode, branch_mode=rule, find_all=True)
    assert want["found"] and want["best"] == 1171 and want["decomposed"] > 1000 and want["leaves"] > 0
    with pb.Engine(p, pb.Config(boundingMode=mode, findAll=True, nbIVMs=4096, **opt)) as e:
        got = e.solve(ub=1171)
    assert got["complete"] and got["found"] and got["cost"] == 1171
    for k in KEYS:
        assert got[k] == want[k], (k, got[k], want[k])
