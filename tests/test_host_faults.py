"""The library's host code on a fake CUDA runtime (tests/fake_cuda.cpp), where
calls can be made to fail and a device can be reset without a GPU."""
import ctypes
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

import pbbperm_b200 as pb

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pbbperm_b200", "csrc")
i32p = ctypes.POINTER(ctypes.c_int32)


@pytest.fixture(scope="session")
def fake_so(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    # -Bsymbolic: the fake runtime is this library's alone
    subprocess.check_call(["g++", "-w", "-shared", "-fPIC", "-O1", "-std=c++17", "-Wl,-Bsymbolic",
                           "-I", "/usr/local/cuda/include", "-I", CSRC, "-o", so, "-x", "c++",
                           *[os.path.join(CSRC, f) for f in ("pbb_host.cu", "pbb_mem.cu", "pbb_pool.cu")],
                           os.path.join(ROOT, "tests", "fake_cuda.cpp"), "-lpthread"])
    return so


@pytest.fixture
def L(fake_so, tmp_path):
    # a library of its own for every test: its state starts empty
    so = str(tmp_path / "libfake.so")
    shutil.copy(fake_so, so)
    lib = ctypes.CDLL(so)
    lib.fake_capacity.argtypes = [ctypes.c_size_t]
    lib.fake_used.restype = ctypes.c_size_t
    lib.pbb_last_error.restype = ctypes.c_char_p
    lib.pbb_engine_destroy.argtypes = [ctypes.c_void_p]
    lib.pbb_start.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p]
    lib.pbb_pool_submit.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p,
                                    ctypes.c_int64]
    lib.pbb_pool_step.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    lib.pbb_pool_destroy.argtypes = [ctypes.c_void_p]
    lib.pbb_get_intervals.argtypes = [ctypes.c_void_p, ctypes.c_int32, i32p, i32p, i32p, ctypes.c_void_p]
    lib.pbb_explore.argtypes = [ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p]
    return lib


def instance(seed, n, m):
    p = np.random.default_rng(seed).integers(1, 99, size=(m, n), dtype=np.int32)
    return pb._instance(p)


def create(L, n=50, m=20, seed=0, **cfg):
    inst, keep = instance(seed, n, m)
    e = ctypes.c_void_p()
    rc = L.pbb_engine_create(ctypes.byref(inst), ctypes.byref(pb.Config(**cfg)._c()), ctypes.byref(e))
    return rc, e


def test_blocks_of_an_engine_that_outlives_its_context_are_not_handed_on(L):
    """A device reset takes all handles with it: an engine destroyed after it
    gives nothing back, and leaves the blocks and streams of engines made since
    alone although they may stand at the same addresses."""
    rc, old = create(L, nbIVMs=65536)                 # over 256 MiB: a block of its own
    assert rc == 0
    L.fake_reset()
    rc, new = create(L, nbIVMs=65536)
    assert rc == 0
    L.pbb_engine_destroy(old)
    rc, third = create(L, nbIVMs=65536)
    assert rc == 0
    assert L.pbb_start(new, 1000, None) == 0 and L.pbb_start(third, 1000, None) == 0
    L.pbb_engine_destroy(new)
    L.pbb_engine_destroy(third)
    rc, again = create(L, nbIVMs=65536)               # from what was kept
    assert rc == 0
    L.pbb_engine_destroy(again)
    assert L.fake_invalid() == 0


def test_nothing_of_a_reset_device_is_used_by_an_engine_made_before(L):
    rc, old = create(L, n=12, m=10, nbIVMs=64)
    assert rc == 0
    L.fake_reset()
    L.pbb_engine_destroy(old)
    rc, new = create(L, n=12, m=10, nbIVMs=64)
    assert rc == 0 and L.pbb_start(new, 1000, None) == 0
    L.pbb_engine_destroy(new)
    assert L.fake_invalid() == 0


def test_streams_are_used_again(L):
    """A stream comes back with its user's frees still on it, and serves the next."""
    for _ in range(20):
        rc, a = create(L, n=12, m=10, nbIVMs=64)
        assert rc == 0
        rc, b = create(L, n=12, m=10, nbIVMs=64)
        assert rc == 0
        L.pbb_engine_destroy(a)
        L.pbb_engine_destroy(b)
    assert L.fake_streams() == 2 and L.fake_invalid() == 0


def bound_call(L, seed, n, m, count, outs=9):
    """pbb_bound_children_ex: (code, outputs)."""
    inst, keep = instance(seed, n, m)
    rng = np.random.default_rng(seed)
    sched = np.argsort(rng.random((count, n)), axis=1).astype(np.int32)
    l1 = rng.integers(-1, n // 2, size=count).astype(np.int32)
    l2 = (l1 + 1 + rng.integers(1, n // 2, size=count)).astype(np.int32)
    arrays = [np.full((count, n) if q < 4 or q in (6, 7) else count, -5, np.int32) for q in range(outs)]
    ptrs = (i32p * 9)(*[a.ctypes.data_as(i32p) for a in arrays])
    rc = L.pbb_bound_children_ex(ctypes.byref(inst), 0, 0, count, sched.ctypes.data_as(i32p), l1.ctypes.data_as(i32p),
                                 l2.ctypes.data_as(i32p), ptrs)
    return rc, arrays


@pytest.mark.parametrize("count", [5, 4000])
def test_every_failed_copy_of_a_bound_call_is_reported(L, count):
    """Inputs that did not arrive are never bounded with what the last call left."""
    L.fake_calls.restype = ctypes.c_int
    assert bound_call(L, 1, 20, 10, count)[0] == 0
    before = L.fake_calls(b"cudaMemcpyAsync")
    rc, want = bound_call(L, 2, 20, 10, count)
    copies = L.fake_calls(b"cudaMemcpyAsync") - before
    assert rc == 0 and copies >= 3 and (want[0] != -5).all()
    for k in range(1, copies + 1):
        assert bound_call(L, 1, 20, 10, count)[0] == 0
        L.fake_fail(b"cudaMemcpyAsync", k)
        assert bound_call(L, 2, 20, 10, count)[0] == pb.PBB_E_CUDA, k
    rc, got = bound_call(L, 2, 20, 10, count)
    assert rc == 0 and all((a == b).all() for a, b in zip(got, want))
    assert L.fake_invalid() == 0


@pytest.mark.parametrize("per_sm,opt,variant", [
    ({}, {}, 3), ({}, dict(adaptiveBranchingMode=2), 4),
    ({4: 1}, {}, 3), ({4: 1}, dict(adaptiveBranchingMode=2), 0), ({3: 1}, {}, 0),
])
def test_pool_windows_launch_only_resident_ctas(L, per_sm, opt, variant):
    """Every build a window launches holds all the CTAs of the pool's grid."""
    for v, c in per_sm.items():
        L.fake_per_sm(v, c)
    inst, keep = instance(1, 12, 10)
    pool = ctypes.c_void_p()
    cfg = pb.PoolConfig(max_jobs=12, max_machines=10, max_resident=2, explorers_per_instance=64)._c()
    assert L.pbb_pool_create(ctypes.byref(cfg), ctypes.byref(pool)) == 0, L.pbb_last_error()
    search = pb.Config(**opt)._c()
    assert L.pbb_pool_submit(pool, ctypes.byref(inst), ctypes.byref(search), 1000, None, 0) == 0
    assert L.pbb_pool_step(pool, None, None) == 0, L.pbb_last_error()
    assert L.fake_variant() == variant and L.fake_not_resident() == 0
    L.pbb_pool_destroy(pool)


def test_an_engine_does_without_pair_bounds_before_it_fails(L):
    """50x20: 95 MB of explorers and 182 MB of pair bounds by level.  With room
    for the explorers alone the general build runs; with less nothing does."""
    L.fake_capacity(200 << 20)
    rc, e = create(L, nbIVMs=4096)
    assert rc == 0, L.pbb_last_error()
    assert L.pbb_start(e, 1000, None) == 0 and L.pbb_explore(e, 1.0, None) == 0
    assert L.fake_variant() == 0
    L.pbb_engine_destroy(e)
    L.fake_capacity(300 << 20)
    rc, e = create(L, nbIVMs=4096)
    assert rc == 0 and L.pbb_start(e, 1000, None) == 0 and L.pbb_explore(e, 1.0, None) == 0
    assert L.fake_variant() == 5
    L.pbb_engine_destroy(e)
    L.fake_capacity(80 << 20)
    assert create(L, nbIVMs=4096)[0] == pb.PBB_E_NOMEM
    L.fake_capacity(300 << 20)
    rc, e = create(L, nbIVMs=4096)
    assert rc == 0
    L.pbb_engine_destroy(e)
    assert L.fake_invalid() == 0


def test_a_pool_does_without_pair_bounds_before_it_fails(L):
    """50x20, two slots: 186 MB of explorers, 91 MB of pair bounds for 2368 warps."""
    inst, keep = instance(1, 50, 20)
    for capacity, variant in ((240, 0), (400, 3)):
        L.fake_capacity(capacity << 20)
        pool = ctypes.c_void_p()
        cfg = pb.PoolConfig(max_jobs=50, max_machines=20, max_resident=2, explorers_per_instance=4096, tail_warps=-1)._c()
        assert L.pbb_pool_create(ctypes.byref(cfg), ctypes.byref(pool)) == 0, L.pbb_last_error()
        search = pb.Config()._c()
        assert L.pbb_pool_submit(pool, ctypes.byref(inst), ctypes.byref(search), 1000, None, 0) == 0
        assert L.pbb_pool_step(pool, None, None) == 0, L.pbb_last_error()
        assert L.fake_variant() == variant
        L.pbb_pool_destroy(pool)
    assert L.fake_invalid() == 0


def test_kept_memory_and_streams_are_released_when_asked_for(L):
    for ivms in (64, 65536, 64):
        rc, e = create(L, nbIVMs=ivms)
        assert rc == 0
        L.pbb_engine_destroy(e)
    rc, e = create(L, nbIVMs=64)
    assert rc == 0
    kept = L.fake_used()
    assert L.pbb_release_memory(0) == 0
    assert 0 < L.fake_used() < kept and L.fake_streams() == 1       # the engine's own
    assert L.pbb_start(e, 1000, None) == 0 and L.pbb_explore(e, 1.0, None) == 0
    L.pbb_engine_destroy(e)
    assert L.pbb_release_memory(0) == 0
    assert L.fake_used() == 0 and L.fake_streams() == 0 and L.fake_invalid() == 0


def test_kept_memory_goes_back_before_sampling_or_a_window_fails(L):
    """Whatever of the library needs memory gets what the library only keeps."""
    rc, old = create(L, nbIVMs=65536)
    assert rc == 0
    rc, e = create(L, n=12, m=10, nbIVMs=64)
    assert rc == 0
    L.pbb_engine_destroy(old)                         # 1.6 GB kept
    L.fake_capacity(L.fake_used() + (1 << 20))
    assert L.pbb_diag_sample_nodes(ctypes.c_void_p(e.value), 100000, 0) == 0, L.pbb_last_error()
    L.pbb_engine_destroy(e)
    L.fake_capacity(1 << 40)
    inst, keep = instance(1, 12, 10)
    pool = ctypes.c_void_p()
    cfg = pb.PoolConfig(max_jobs=12, max_machines=10, max_resident=2, explorers_per_instance=64)._c()
    assert L.pbb_pool_create(ctypes.byref(cfg), ctypes.byref(pool)) == 0, L.pbb_last_error()
    search = pb.Config()._c()
    assert L.pbb_pool_submit(pool, ctypes.byref(inst), ctypes.byref(search), 1000, None, 0) == 0
    L.fake_fail(b"cudaGraphInstantiate", 1)
    assert L.pbb_pool_step(pool, None, None) == 0, L.pbb_last_error()
    L.pbb_pool_destroy(pool)
    assert L.fake_invalid() == 0


def test_threads_share_what_is_kept(L):
    """Engines and bound calls of several sizes from eight threads at once: no
    block or stream is lent twice or after it went back."""
    bad = []

    def work(t):
        for i in range(12):
            rc, e = create(L, n=(12, 50)[(t + i) % 2], m=(10, 20)[(t + i) % 2], nbIVMs=(64, 12000)[(t + i) % 2])
            if rc or L.pbb_start(e, 1000, None) or L.pbb_explore(e, 1.0, None):
                bad.append((t, i))
            rc, out = bound_call(L, t, 20, 10, (5, 3000)[i % 2])
            want = bound_call(L, t, 20, 10, (5, 3000)[i % 2])[1]
            if rc or any((a != b).any() for a, b in zip(out, want)):
                bad.append((t, i, "bounds"))
            L.pbb_engine_destroy(e)
            if i == 6:
                L.pbb_release_memory(0)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad and L.fake_invalid() == 0
    assert L.pbb_release_memory(0) == 0
    assert L.fake_used() == 0 and L.fake_streams() == 0


def test_short_windows_share_fully_unless_their_caller_exports(L):
    """Under 5 ms, the first window and one after an export keep the number of
    intervals down; other windows do not."""
    L.fake_windows(100)
    rc, e = create(L, n=12, m=10, nbIVMs=64)
    assert rc == 0
    pos, end, ids = (np.zeros(64 * 12, np.int32) for _ in range(3))
    cnt = ctypes.c_int32()

    def window(seconds):
        assert L.pbb_explore(e, seconds, None) == 0
        return L.fake_eager()

    for _ in range(2):
        assert L.pbb_start(e, 1000, None) == 0
        assert [window(0.002), window(0.002), window(0.002)] == [0, 1, 1]
        assert L.pbb_get_intervals(e, 64, pos.ctypes.data_as(i32p), end.ctypes.data_as(i32p), ids.ctypes.data_as(i32p),
                                   ctypes.byref(cnt)) == 0
        assert [window(0.002), window(0.002)] == [0, 1]
        assert L.pbb_start(e, 1000, None) == 0
        assert [window(0.006), window(0.001)] == [1, 1]
    L.pbb_engine_destroy(e)
