"""The work a user has this framework do, as cases that can be timed.

Kinds of case:

  search  one branch-and-bound search to completion through pb.Engine
  batch   many instances solved from NEH through one resident pool
          (pb.batch_solve, or pb.Pool driven by the caller)
  bounds  children bounds of a batch of nodes: host arrays through
          pb.bound_children(_ex), or device buffers through the no-alloc entry
  neh     NEH of many instances on the device
  ig      iterated greedy of many instances on the device

Searches start from a target no schedule beats (the optimum, or a lower value
whose proof fits the time), as the reference's own parity runs do: nothing
improves on it, so the decomposed-node counts are those of the instance and
not of the order in which explorers met.  The catalogue below holds base
instances of the project's generator with such targets; a case's input is a
base instance with its jobs in another order and one processing time in a
hundred one unit longer, which can only raise the optimum.
"""
import ctypes
import math

import numpy as np
import torch

import pbbperm_b200 as pb
from pbbperm_b200.instances import synthetic_instance

# (bounding mode, branching rule, jobs, machines, instance seed, target,
#  decomposed nodes, one-machine bounds, Johnson bounds) of the base instance
CATALOGUE = [
    (2, 3, 12, 10, 1, 1180, 953, 11856, 1668),
    (2, 3, 12, 10, 2, 1238, 588, 8712, 1170),
    (2, 3, 12, 10, 3, 1171, 1712, 20162, 3105),
    (2, 3, 14, 10, 1, 1221, 1436, 20484, 2652),
    (2, 3, 14, 10, 2, 1304, 3041, 45848, 10080),
    (2, 3, 14, 10, 3, 1218, 580, 7986, 824),
    (2, 3, 14, 20, 1, 1915, 18563, 279966, 57394),
    (2, 3, 14, 20, 2, 1949, 60056, 856612, 149839),
    (2, 3, 14, 20, 3, 1881, 184819, 2534898, 363401),
    (2, 3, 16, 10, 1, 1312, 4987, 66732, 6749),
    (2, 3, 16, 10, 2, 1392, 4457, 72586, 6155),
    (2, 3, 16, 10, 3, 1387, 38767, 604812, 102039),
    (2, 3, 16, 20, 1, 2039, 86397, 1486550, 133290),
    (2, 3, 16, 20, 2, 2087, 619487, 9640772, 1184138),
    (2, 3, 16, 20, 3, 2081, 1850798, 26117446, 6399555),
    (2, 3, 18, 10, 2, 1527, 2519, 39544, 3359),
    (2, 3, 18, 20, 1, 2150, 571457, 10513802, 1101215),
    (2, 3, 18, 20, 2, 2229, 872540, 17475400, 2445987),
    (2, 3, 18, 20, 3, 2178, 19098299, 327908954, 43057088),
    (2, 3, 20, 10, 1, 1548, 2620, 45638, 3358),
    (2, 3, 20, 10, 2, 1590, 7022, 161704, 9913),
    (2, 3, 20, 10, 3, 1528, 119942, 2436838, 180104),
    (2, 3, 20, 20, 1, 2352, 12616547, 236462768, 25431709),
    (2, 3, 20, 20, 3, 2210, 12167926, 235209100, 19862266),
    (2, 3, 24, 10, 1, 1833, 5033, 143290, 6297),
    (2, 3, 24, 10, 2, 1792, 2363, 55900, 3081),
    (2, 3, 24, 10, 3, 1721, 489961, 11375222, 600496),
    (2, 3, 25, 20, 1, 2468, 2556247, 77811396, 3275689),
    (2, 3, 30, 10, 2, 2137, 10488101, 306700620, 14604649),
    (2, 3, 30, 10, 3, 2005, 99391, 3217528, 114620),
    (2, 3, 30, 20, 3, 2654, 54473483, 1975739920, 69111651),
    (2, 3, 33, 15, 2, 2536, 47599807, 1438898250, 53005743),
    (2, 3, 33, 15, 3, 2436, 34741162, 1304165080, 37462916),
    (2, 3, 40, 10, 3, 2494, 293047, 12391668, 324651),
    (2, 3, 40, 20, 3, 3136, 59917815, 3018409272, 67604187),
    (2, 3, 50, 20, 3, 3673, 55883197, 4210935954, 66626960),
    (0, 2, 13, 10, 3, 1277, 8390, 110600, 0),
    (0, 2, 14, 20, 2, 1949, 404545, 4553936, 0),
    (0, 2, 15, 10, 3, 1364, 44551, 569912, 0),
    (0, 2, 17, 10, 2, 1457, 14434, 246460, 0),
    (0, 2, 18, 20, 2, 2229, 9601904, 159584150, 0),
    (0, 2, 20, 10, 3, 1528, 189748, 3444508, 0),
    (0, 2, 20, 20, 3, 2210, 26783972, 479497368, 0),
    (0, 2, 25, 10, 3, 1797, 4136214, 83808312, 0),
    (0, 2, 30, 10, 3, 2005, 104345, 3393440, 0),
    (0, 2, 30, 20, 3, 2645, 27237427, 1017355390, 0),
    (0, 2, 40, 20, 3, 3131, 25990871, 1337998598, 0),
    (0, 2, 50, 20, 3, 3666, 26112834, 1995091318, 0),
    (0, 3, 13, 10, 3, 1277, 6801, 90962, 0),
    (0, 3, 14, 20, 2, 1949, 424916, 4860472, 0),
    (0, 3, 15, 10, 3, 1364, 46225, 593320, 0),
    (0, 3, 17, 10, 2, 1457, 14044, 239808, 0),
    (0, 3, 18, 20, 2, 2229, 8805445, 146289488, 0),
    (0, 3, 20, 10, 3, 1528, 216107, 3975982, 0),
    (0, 3, 20, 20, 3, 2210, 25609733, 462477982, 0),
    (0, 3, 25, 10, 3, 1797, 3605394, 74494500, 0),
    (0, 3, 30, 10, 3, 2005, 116662, 3715078, 0),
    (0, 3, 30, 20, 3, 2646, 28276870, 1052141498, 0),
    (0, 3, 40, 20, 3, 3131, 27313539, 1407694358, 0),
    (0, 3, 50, 20, 3, 3667, 29977165, 2282473504, 0),
    (1, 2, 13, 10, 3, 1277, 1529, 0, 23196),
    (1, 2, 14, 20, 2, 1949, 9482, 0, 146694),
    (1, 2, 15, 10, 3, 1364, 22663, 0, 320274),
    (1, 2, 17, 10, 2, 1457, 4945, 0, 90852),
    (1, 2, 18, 20, 2, 2229, 634514, 0, 12963838),
    (1, 2, 20, 10, 3, 1528, 90379, 0, 1842022),
    (1, 2, 20, 20, 3, 2210, 11576310, 0, 223738936),
    (1, 2, 25, 10, 3, 1797, 2839640, 0, 62235080),
    (1, 2, 30, 10, 3, 2005, 83197, 0, 2770480),
    (1, 3, 13, 10, 3, 1277, 1234, 0, 18932),
    (1, 3, 14, 20, 2, 1949, 27669, 0, 434442),
    (1, 3, 15, 10, 3, 1364, 24075, 0, 344900),
    (1, 3, 17, 10, 2, 1457, 3663, 0, 66878),
    (1, 3, 18, 20, 2, 2229, 632030, 0, 13051620),
    (1, 3, 20, 10, 3, 1528, 95664, 0, 1937784),
    (1, 3, 20, 20, 3, 2210, 10950654, 0, 216806334),
    (1, 3, 25, 10, 3, 1797, 2490506, 0, 54936154),
    (1, 3, 30, 10, 3, 2005, 91646, 0, 3014360),
    (2, 1, 13, 10, 3, 1277, 2404, 36064, 5418),
    (2, 1, 14, 20, 2, 1949, 79913, 1069970, 177591),
    (2, 1, 15, 10, 3, 1364, 31296, 424102, 45770),
    (2, 1, 17, 10, 2, 1457, 8162, 144138, 13649),
    (2, 1, 18, 20, 2, 2229, 1104239, 21339366, 3007177),
    (2, 1, 20, 10, 3, 1528, 122257, 2396310, 190271),
    (2, 1, 20, 20, 3, 2210, 18285886, 337632758, 27542255),
    (2, 1, 25, 10, 3, 1797, 2380607, 51162796, 2989313),
    (2, 1, 30, 10, 3, 2005, 128871, 4039178, 146981),
    (2, 1, 30, 20, 3, 2646, 28935096, 1075792834, 37188651),
    (2, 1, 40, 20, 3, 3131, 27620643, 1418094852, 32169449),
    (2, 1, 50, 20, 3, 3666, 26541107, 2018594600, 32801044),
    (2, 2, 13, 10, 3, 1277, 2238, 33618, 5031),
    (2, 2, 14, 20, 2, 1949, 70169, 968304, 162443),
    (2, 2, 15, 10, 3, 1364, 27201, 374740, 39951),
    (2, 2, 17, 10, 2, 1457, 7133, 127718, 11909),
    (2, 2, 18, 20, 2, 2229, 1039331, 20379484, 2811355),
    (2, 2, 20, 10, 3, 1528, 104804, 2107710, 157770),
    (2, 2, 20, 20, 3, 2210, 14537372, 274513918, 22264464),
    (2, 2, 25, 10, 3, 1797, 3026027, 64899320, 3812874),
    (2, 2, 30, 10, 3, 2005, 88679, 2922140, 102934),
    (2, 2, 30, 20, 3, 2647, 27276924, 1016627532, 34013291),
    (2, 2, 40, 20, 3, 3132, 26964294, 1383220418, 30624616),
    (2, 2, 50, 20, 3, 3668, 29049275, 2209776256, 34831861),
]
ROW = {r[:5]: r for r in CATALOGUE}


def _search(name, mode, rule, n, m, inst, ivms=16384, fresh=False, sort=0, early=False, parts=0):
    return dict(name=name, kind="search", mode=mode, rule=rule, n=n, m=m, inst=inst, ivms=ivms, fresh=fresh, sort=sort,
                early=early, parts=parts)


def listed():
    return [
        # the smallest whole calls: a new engine, a search of about a thousand nodes, the result
        _search("solve_12x10", 2, 3, 12, 10, 3, fresh=True),
        # an ordinary whole call: 20 jobs, 10 machines, about 10^5 nodes
        _search("solve_20x10", 2, 3, 20, 10, 3, fresh=True),
        # the reference's 20x20 optimality proof, default search, 16384 explorers
        _search("prove_20x20", 2, 3, 20, 20, 1),
        # the headline shape: 50 jobs, 20 machines, 65536 explorers
        _search("prove_50x20", 2, 3, 50, 20, 3, ivms=65536),
        # Johnson bound on every child, sorted rows, early exit: the other options people set in gpuconfig.ini
        _search("johnson_sorted_20x20", 1, 2, 20, 20, 3, sort=1, early=True),
        # one-machine bound alone
        _search("weak_18x20", 0, 3, 18, 20, 2),
        # a batch of uneven instances from their NEH bounds, whole call
        dict(name="batch_64_mixed", kind="batch", count=64, nlo=10, nhi=16, api="batch"),
        # bounds library calls: a handful of nodes (a CPU search asking for its children), and a big batch with priorities
        dict(name="bounds_64_20x20", kind="bounds", count=64, n=20, m=20, jmode=0, api="host"),
        dict(name="bounds_20000_50x20_ex", kind="bounds", count=20000, n=50, m=20, jmode=0, api="host_ex"),
        # the same library from a program that keeps its nodes on the GPU
        dict(name="bounds_50000_50x20_device", kind="bounds", count=50000, n=50, m=20, jmode=0, api="device"),
        # starting bounds of a batch of requests
        dict(name="neh_512_mixed", kind="neh", count=512, nlo=12, nhi=22, m=20),
        # better starting bounds for large instances
        dict(name="ig_64_50x20", kind="ig", count=64, nlo=50, nhi=50, m=20, iterations=5),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["batch", "bounds", "bounds", "bounds", "neh", "ig"])
    if kind == "search":
        default = [r for r in CATALOGUE if r[:2] == (2, 3)]
        others = [r for r in CATALOGUE if r[:2] != (2, 3)]
        row = rng.choice(default if rng.random() < 0.6 else others)
        mode, rule, n, m, inst = row[:5]
        big = row[6] > 2e7      # the longest proofs: as the listed ones run them
        c = _search("", mode, rule, n, m, inst, ivms=rng.choice([16384, 32768, 65536] + [4096] * (not big)),
                    fresh=rng.random() < 0.5, sort=0 if big else rng.choice([0, 0, 0, 1]),
                    early=not big and rng.random() < 0.25, parts=rng.choice([0, 0, 0, 0, 7, 100]))
    elif kind == "batch":
        lo = rng.randint(8, 12)
        c = dict(kind="batch", count=_log_int(rng, 3, 80), nlo=lo, nhi=lo + rng.randint(0, 4),
                 api=rng.choice(["batch", "pool"]))
    elif kind == "bounds":
        c = dict(kind="bounds", count=_log_int(rng, 1, 40000), n=rng.randint(8, 60), m=rng.randint(3, 20),
                 jmode=rng.choice([0, 0, 0, 1, 2]), api=rng.choice(["host", "host", "host_ex", "device", "device"]))
        if c["api"] == "host_ex":
            c["count"] = min(c["count"], 20000)
    elif kind == "neh":
        lo = rng.randint(6, 55)
        c = dict(kind="neh", count=_log_int(rng, 1, 512), nlo=lo, nhi=min(64, lo + rng.randint(0, 12)),
                 m=rng.randint(3, 20))
    else:
        lo = rng.randint(6, 46)
        c = dict(kind="ig", count=_log_int(rng, 1, 128), nlo=lo, nhi=lo + rng.randint(0, 4), m=rng.randint(3, 20),
                 iterations=rng.randint(1, 5))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _base(case, seed):
    """The case's base instance, jobs reordered, some times one unit longer."""
    rng = np.random.default_rng(seed)
    p = synthetic_instance(case["inst"], case["n"], case["m"])[:, rng.permutation(case["n"])].copy()
    grown = rng.choice(p.size, max(2, p.size // 100), replace=False)
    p.reshape(-1)[grown] += 1
    return p


def _instances(rng, count, nlo, nhi, machines):
    out = []
    for _ in range(count):
        n = int(rng.integers(nlo, nhi + 1))
        m = int(rng.choice(machines))
        out.append(rng.integers(1, 100, size=(m, n)).astype(np.int32))
    return out


def _nodes(rng, n, count):
    """Nodes of every depth: k free jobs (1..n), the rest split between the
    front and the back."""
    sched = np.argsort(rng.random((count, n)), axis=1).astype(np.int32)
    k = rng.integers(1, n + 1, size=count)
    front = (rng.random(count) * (n - k + 1)).astype(np.int64)
    return sched, (front - 1).astype(np.int32), (front + k).astype(np.int32)


def _split_root(n, parts):
    """The whole permutation space as `parts` factoradic intervals."""
    total = math.factorial(n)

    def digits(x):
        d = [0] * n
        for i in range(n - 1, -1, -1):
            x, d[i] = divmod(x, n - i)
        return d

    cuts = [total * i // parts for i in range(parts + 1)]
    pos = np.array([digits(cuts[i]) for i in range(parts)], np.int32)
    end = np.array([digits(cuts[i + 1] - 1) for i in range(parts)], np.int32)
    return pos, end


def _engine(case, p):
    return pb.Engine(p, pb.Config(boundingMode=case["mode"], adaptiveBranchingMode=case["rule"], nbIVMs=case["ivms"],
                                  sortedDFS=case["sort"], earlyStopJohnson=case["early"]))


def _row(case):
    return ROW[(case["mode"], case["rule"], case["n"], case["m"], case["inst"])]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "search":
        s["p"] = _base(case, seed)
        s["target"] = _row(case)[5]
        if case["parts"]:
            s["pos"], s["end"] = _split_root(case["n"], case["parts"])
        if not case["fresh"]:
            s["engine"] = _engine(case, s["p"])
    elif kind == "batch":
        s["inst"] = _instances(rng, case["count"], case["nlo"], case["nhi"], (5, 10, 20))
        if case["api"] == "pool":
            s["pool"] = pb.Pool(pb.PoolConfig(max_jobs=case["nhi"], max_machines=20, window_s=0.002))
    elif kind == "bounds":
        s["p"] = rng.integers(1, 100, size=(case["m"], case["n"])).astype(np.int32)
        s["sched"], s["l1"], s["l2"] = _nodes(rng, case["n"], case["count"])
        if case["api"] == "device":
            dev = torch.device("cuda")
            s["dev"] = [torch.from_numpy(a).to(dev) for a in (s["sched"], s["l1"], s["l2"])]
            s["out"] = [torch.zeros((case["count"], case["n"]), dtype=torch.int32, device=dev) for _ in range(4)]
            s["out"] += [torch.zeros(case["count"], dtype=torch.int32, device=dev) for _ in range(2)]
    else:
        s["inst"] = _instances(rng, case["count"], case["nlo"], case["nhi"], (case["m"],))
        s["seed"] = seed
    return s


# ---------------------------------------------------------------------------
# passes
# ---------------------------------------------------------------------------
def _run_search(s, engine):
    if "pos" in s:
        engine.init_from_fac(s["target"], s["pos"], s["end"])
        done = False
        while not done:
            done = engine.explore(2.0)
        r = engine.result()
    else:
        r = engine.solve(ub=s["target"])
    # the counts of a proof: nothing improves on the target, so they do not
    # depend on the order of the exploration
    return {k: r[k] for k in ("complete", "found", "cost", "decomposed", "simple_bounds", "johnson_bounds", "leaves")}


def _run_device_bounds(s):
    p = s["p"]
    m, n = p.shape
    i32p = ctypes.POINTER(ctypes.c_int32)
    inst = pb._Instance(n, m, p.ctypes.data_as(i32p))
    fn = pb.lib().pbb_bound_children_noalloc
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in s["dev"] + s["out"]]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    pb._check(fn(ctypes.byref(inst), ctypes.c_int32(s["case"]["jmode"]), ctypes.c_int32(torch.cuda.current_device()),
                 stream, ctypes.c_int32(len(s["sched"])), *ptr))
    return s["out"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "search":
        if not case["fresh"]:
            return _run_search(state, state["engine"])
        with _engine(case, state["p"]) as engine:
            return _run_search(state, engine)
    if kind == "batch":
        inst = state["inst"]
        cost = np.zeros(len(inst), np.int32)
        if case["api"] == "batch":
            # which optimal schedule is found first is not determined; its makespan is
            for i, r in enumerate(pb.batch_solve(inst, ubs=[pb.UB_NEH] * len(inst))):
                cost[i] = r["cost"]
        else:
            pool = state["pool"]
            for i, p in enumerate(inst):
                pool.submit(p, tag=i, ub=pb.UB_NEH)
            left = len(inst)
            while left:
                pool.step()
                for r in pool.poll():
                    cost[r["tag"]] = r["cost"]
                    left -= 1
        return cost
    if kind == "bounds":
        if case["api"] == "device":
            return _run_device_bounds(state)
        fn = pb.bound_children_ex if case["api"] == "host_ex" else pb.bound_children
        return fn(state["p"], state["sched"], state["l1"], state["l2"], johnson_mode=case["jmode"])
    if kind == "neh":
        res = pb.neh_batch(state["inst"])
    else:
        res = pb.ig_batch(state["inst"], iterations=case["iterations"], seed=state["seed"])
    return _schedules(res, case["nhi"])


def _schedules(res, width):
    """(cost, schedule) pairs as two arrays, schedules padded with -1."""
    perms = np.full((len(res), width), -1, np.int32)
    for row, (_, q) in zip(perms, res):
        row[:len(q)] = q
    return [np.array([c for c, _ in res], np.int32), perms]


# ---------------------------------------------------------------------------
# work a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "search":
        # 5 operations per machine of a one-machine bound; per Johnson bound
        # at least one add, one max and one compare for every machine pair
        m = case["m"]
        _, _, n, _, _, _, nodes, simple, johnson = _row(case)
        return dict(bytes=4 * n * m + 8 * n, flops=5 * m * simple + 3 * (m * (m - 1) // 2) * johnson + 10 * nodes)
    if kind == "batch":
        n = (case["nlo"] + case["nhi"]) / 2
        return dict(bytes=case["count"] * n * 4 * 12, flops=case["count"] * 40.0 * n ** 4)
    if kind == "bounds":
        n, m, cnt = case["n"], case["m"], case["count"]
        pairs = {0: m * (m - 1) // 2, 1: m - 1, 2: m - 1}[case["jmode"]]
        k = (n + 1) / 2
        words = cnt * (5 * n + 4) + (cnt * (2 * n + 1) if case["api"] == "host_ex" else 0)
        # one-machine bounds of 2k children; per pair two max-plus passes over the k free jobs, and each child from them
        return dict(bytes=4.0 * words, flops=cnt * (2 * k * 5 * m + pairs * (10 * k + 2 * k * 5)))
    n = (case["nlo"] + case["nhi"]) / 2
    insert = 3 * n * case["m"] * 2 + n * case["m"] * 4     # heads, tails, and every position of one insertion
    rounds = n / 2 if kind == "neh" else n / 2 + case["iterations"] * (3 + 2 * n)
    return dict(bytes=case["count"] * 4.0 * (n * case["m"] + n + 1), flops=case["count"] * rounds * insert)


# ---------------------------------------------------------------------------
# the same values by plain numpy in 64 bits
# ---------------------------------------------------------------------------
def _johnson_order(pa, pb_, lag):
    """Johnson's order with lags; ties as a quicksort with Hoare's partition
    around the first element leaves them (part of the bound's definition)."""
    first = pa < pb_
    key = [(0, pa[j] + lag[j]) if first[j] else (1, -(pb_[j] + lag[j])) for j in range(len(pa))]
    v = list(range(len(pa)))

    def sort(lo, hi):
        if lo >= hi:
            return
        pivot, i, j = key[v[lo]], lo - 1, hi + 1
        while True:
            j -= 1
            while key[v[j]] > pivot:
                j -= 1
            i += 1
            while key[v[i]] < pivot:
                i += 1
            if i >= j:
                break
            v[i], v[j] = v[j], v[i]
        sort(lo, j)
        sort(j + 1, hi)

    sort(0, len(v) - 1)
    return v


def _heads(p, seq, start=None):
    h = np.zeros(p.shape[0], np.int64) if start is None else start.copy()
    for j in seq:
        t = 0
        for k in range(len(h)):
            h[k] = t = max(h[k], t) + p[k, j]
    return h


def _exact_bounds(case, seed):
    s = prepare(dict(case, api="host"), seed)
    p = s["p"].astype(np.int64)
    m, n = p.shape
    mode = case["jmode"]
    pairs = [(a, b) for a in range(m) for b in range(a + 1, m)
             if mode == 0 or (mode == 1 and b == m - 1) or (mode == 2 and b == a + 1)]
    a, b = np.array([x for x, _ in pairs]), np.array([y for _, y in pairs])
    lag = np.array([[p[x + 1:y, j].sum() for j in range(n)] for x, y in pairs])
    order = np.array([_johnson_order(p[x], p[y], lag[i]) for i, (x, y) in enumerate(pairs)])
    arrive = np.array([min(p[:k, j].sum() for j in range(n)) for k in range(m)])
    depart = np.array([min(p[k + 1:, j].sum() for j in range(n)) for k in range(m)])
    idx = np.arange(len(pairs))

    def johnson(front, back, free):
        """front, back: heads and tails; free: boolean by job."""
        t0, t1 = front[a].copy(), front[b].copy()
        for t in range(n):
            j = order[:, t]
            on = free[j]
            x0 = t0 + p[a, j]
            x1 = np.maximum(t1, x0 + lag[idx, j]) + p[b, j]
            t0, t1 = np.where(on, x0, t0), np.where(on, x1, t1)
        return int(np.maximum(t1 + back[b], t0 + back[a]).max())

    def span(seq):
        return int(_heads(p, seq)[-1])

    def tails(seq):
        return _heads(p[::-1], seq[::-1])[::-1]

    def strong(sc, f, e):
        """Johnson value of the node with jobs [0, f) in front, [e, n) behind."""
        if e - f <= 1:
            return span(sc)
        front = _heads(p, sc[:f]) if f else arrive
        back = tails(sc[e:]) if e < n else depart
        free = np.zeros(n, bool)
        free[sc[f:e]] = True
        return johnson(front, back, free)

    cnt = case["count"]
    out = {k: np.zeros((cnt, n), np.int64) for k in ("weak_begin", "weak_end", "strong_begin", "strong_end")}
    out["node_weak"], out["node_strong"] = np.zeros(cnt, np.int64), np.zeros(cnt, np.int64)
    for i in range(cnt):
        sc = [int(x) for x in s["sched"][i]]
        f, e = int(s["l1"][i]) + 1, int(s["l2"][i])
        front = _heads(p, sc[:f]) if f else arrive
        back = tails(sc[e:]) if e < n else depart
        rest = p[:, sc[f:e]].sum(axis=1)
        t, lb = 0, 0
        for k in range(m):
            t = max(front[k] + rest[k], t) if k else front[0] + rest[0]
            lb = max(lb, t + back[k])
        out["node_weak"][i] = lb
        out["node_strong"][i] = strong(sc, f, e)
        for j in sc[f:e]:
            t, lb = 0, 0
            for k in range(m):
                t = max(front[k], t) if k else front[0]
                lb, t = max(lb, t + rest[k] + back[k]), t + p[k, j]
            out["weak_begin"][i, j] = lb
            t, lb = 0, 0
            for k in range(m - 1, -1, -1):
                t = max(back[k], t) if k < m - 1 else back[k]
                lb, t = max(lb, t + rest[k] + front[k]), t + p[k, j]
            out["weak_end"][i, j] = lb
            others = [x for x in sc[f:e] if x != j]
            out["strong_begin"][i, j] = strong(sc[:f] + [j] + others + sc[e:], f + 1, e)
            out["strong_end"][i, j] = strong(sc[:f] + others + [j] + sc[e:], f, e - 1)
    return out


def _exact_neh(case, seed):
    res = []
    for q in prepare(case, seed)["inst"]:
        p = q.astype(np.int64)
        m, n = p.shape
        order = sorted(range(n), key=lambda j: (-p[:, j].sum(), j))
        seq = []
        for x in order:
            spans = []
            for pos in range(len(seq) + 1):
                spans.append(int(_heads(p, seq[:pos] + [x] + seq[pos:])[-1]))
            best = spans.index(min(spans))
            seq.insert(best, x)
        res.append((int(_heads(p, seq)[-1]), seq))
    return _schedules(res, case["nhi"])


def exact(case, seed):
    if case["kind"] == "bounds":
        n, m = case["n"], case["m"]
        if case["api"] != "host" or case["count"] * n * n * (60e-6 + m * m * 2e-7) > 15:
            return None
        return _exact_bounds(case, seed)
    if case["kind"] == "neh":
        if case["count"] * case["nhi"] ** 3 * case["m"] * 2e-7 / 2 > 10:
            return None
        return _exact_neh(case, seed)
    # searches, batches and the seeded local search have no closed form
    return None
