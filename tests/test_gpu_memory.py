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
