"""Work sharing inside and between CTAs: whatever the launch shape (CTAs and
warps with and without explorers of their own, mask words of the asking CTAs
partly used), the window length and the sharing threshold, the counters are
the oracle's."""
import pytest

from oracle import Oracle
import pbbperm_b200 as pb
from pbbperm_b200.instances import synthetic_instance

pytestmark = pytest.mark.gpu

KEYS = ("decomposed", "johnson_bounds", "simple_bounds", "leaves")


@pytest.fixture(scope="module")
def case():
    p = synthetic_instance(3, 12, 10)
    O = Oracle(p)
    return p, 1171, {mode: O.solve(1171, bound_mode=mode) for mode in (0, 2)}


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("ivms,ctas,warps", [(1, 0, 0), (2, 0, 1), (31, 33, 1), (33, 32, 1), (149, 0, 1), (40, 2, 20),
                                             (3000, 0, 0), (700, 65, 7)])
@pytest.mark.parametrize("share_after", [-1, 0, 2**31 - 1])
def test_counts_do_not_depend_on_the_launch_shape(case, mode, ivms, ctas, warps, share_after):
    p, opt, want = case
    cfg = pb.Config(boundingMode=mode, nbIVMs=ivms, ctas=ctas, warps_per_cta=warps, share_after=share_after)
    with pb.Engine(p, cfg) as e:
        got = e.solve(ub=opt)
        again = e.solve(ub=opt)         # requests left by the first search are gone
        e.start(ub=opt)
        while not e.explore(0.0003):    # short windows: intervals carried from launch to launch
            pass
        windows = e.result()
    for r in (got, again, windows):
        assert r["complete"] and not r["found"]
        for k in KEYS:
            assert r[k] == want[mode][k], (k, r[k], want[mode][k])
    if share_after == 2**31 - 1:
        assert got["steals"] == 0
