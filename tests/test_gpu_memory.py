"""Freed device blocks wait for the next index, within a bound, and go back to
the driver on gts_memory_release; indexes built from reused blocks answer as
any other."""
import ctypes as C
import threading

import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


def _release():
    n = C.c_size_t()
    assert gts._load_lib().gts_memory_release(C.byref(n)) == 0
    return n.value


def test_blocks_wait_and_go_back():
    import torch
    rows = G.gmm_rows(200_000, 64, 16, 0.3, seed=1)   # rows and their tree-ordered copy: 51 MB each
    q = G.query_ids(200_000, 200, 2)
    with gts.Index(rows, 2, max_h=5) as idx:
        want = idx.knn(q, 8, return_ids=True)
    _release()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    with gts.Index(rows, 2, max_h=5) as idx:
        idx.knn(q, 8)
    kept = free0 - torch.cuda.mem_get_info()[0]
    assert 100e6 < kept < 4.5e9
    with gts.Index(rows[::-1].copy(), 2, max_h=5):   # other contents in the same blocks
        pass
    with gts.Index(rows, 2, max_h=5) as idx:
        for x, y in zip(idx.knn(q, 8, return_ids=True), want):
            np.testing.assert_array_equal(x, y)
    assert _release() >= 100_000_000
    assert free0 - torch.cuda.mem_get_info()[0] < 32e6
    assert _release() == 0


def test_two_threads_build_and_ask():
    sets = [G.gmm_rows(60_000, 32, 10, 0.3, seed=s) for s in (3, 4)]
    q = G.query_ids(60_000, 100, 5)
    want = []
    for rows in sets:
        with gts.Index(rows, 2, max_h=5) as idx:
            want.append(idx.knn(q, 8))
    bad = []

    def work(i):
        for _ in range(6):
            with gts.Index(sets[i], 2, max_h=5) as idx:
                if not np.array_equal(idx.knn(q, 8), want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_an_index_freed_by_another_thread_gives_its_blocks_back():
    """The freeing thread has made no CUDA call before."""
    import torch
    rows = G.gmm_rows(300_000, 64, 16, 0.3, seed=6)   # 77 MB a copy
    gts.Index(rows[:1000], 2, max_h=2).close()
    _release()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        idx = gts.Index(rows, 2, max_h=5)
        idx.prepare()
        t = threading.Thread(target=idx.close)
        t.start()
        t.join()
    _release()
    assert free0 - torch.cuda.mem_get_info()[0] < 32e6


def _used(call):
    import torch
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    out = call()
    torch.cuda.synchronize()
    return out, free0 - torch.cuda.mem_get_info()[0]


SLACK = 4 << 20   # argument buffers, blocks rounded to 2 MiB


def test_hit_lists_stay_in_the_budget():
    n = 16_000   # a list holds all of them
    rows = G.gmm_rows(n, 32, 1, 1.0, seed=3)
    q = G.query_ids(n, 128, 4)
    r = float(np.float32(G.quantile_radius(2, 0.6, 20000, 5, rows=rows)))
    budget = 22 << 20   # 3 for a tile, 16 for its longer lists, the hits are 10
    with gts.Index(rows, 2, max_h=4) as big, gts.Index(rows, 2, max_h=4, mem_budget_gb=budget / 2**30) as small:
        want = big.range_ids(q, r)
        room = len(want[2])
        assert 8 * room > 9 << 20
        small.range(q[:1], r)
        _release()
        got, used = _used(lambda: small.range_ids(q, r, capacity=room))
        for x, y in zip(got, want):
            np.testing.assert_array_equal(x, y)
        assert used <= budget + SLACK, f"{used >> 20} MiB"


def test_a_stream_and_its_sweep_share_the_budget():
    n = 200_000
    rows = G.gmm_rows(n, 16, 16, 0.3, seed=6)
    ids = G.query_ids(n, 3000, 7)
    flags = np.full(len(ids), 2, np.int32)
    r = float(np.float32(G.quantile_radius(2, 0.05, 20000, 8, rows=rows)))
    budget = 27 << 20   # entries of 4 MB; eight of the sweep's tiles take 25
    with gts.Index(rows, 2, max_h=5) as big, gts.Index(rows, 2, max_h=5, mem_budget_gb=budget / 2**30) as small:
        want = big.update_run(flags, ids, r)[0]
        _release()
        got, used = _used(lambda: small.update_run(flags, ids, r)[0])
        np.testing.assert_array_equal(got, want)
        assert used <= budget, f"{used >> 20} MiB"


def test_small_batches_leave_their_buffers_out_of_a_tight_budget():
    rows = G.gmm_rows(20_000, 32, 16, 0.3, seed=9)
    q = G.query_ids(20_000, 64, 10)

    def launches(budget):
        with gts.Index(rows, 2, max_h=4, mem_budget_gb=budget / 2**30) as idx:
            idx.prepare()
            try:
                kth = idx.knn(q, 8, form=gts.FORM_FAST)
            except gts.GtsError:
                return None, None
            n0 = idx.kernel_launches()
            np.testing.assert_array_equal(idx.knn(q, 8, form=gts.FORM_FAST), kth)
            return idx.kernel_launches() - n0, kth

    ample, want = launches(1 << 30)
    assert ample == 3                          # no tiles
    lo, hi = 1 << 10, 64 << 20                 # the least budget of one run of the tiles
    while hi - lo > 1 << 12:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if launches(mid)[0] else (mid, hi)
    tight, got = launches(hi)
    assert tight > 3
    np.testing.assert_array_equal(got, want)


def test_memory_release_from_python():
    with gts.Index(G.gmm_rows(100_000, 64, 16, 0.3, seed=11), 2, max_h=4):
        pass
    assert gts.memory_release() >= 50_000_000
    assert gts.memory_release() == 0
