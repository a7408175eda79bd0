"""Which of the plain form's searches answers a batch: the one that is chosen
is not slower than the per-query traversal (pinned threads), for few and many
queries, selective and wide radii, small and large leaves; and the answers are
the traversal's on both sides of each line the rules draw."""
import time

import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


def _best_s(call, reps):
    t = []
    for _ in range(reps):
        t0 = time.perf_counter()
        call()
        t.append(time.perf_counter() - t0)
    return min(t)


def _not_slower(auto, pinned, reps=6):
    """Up to 1.5 times and 40 us more pass: launches are a few us each, and
    the faults this looks for were 2 to 20 times.  The best of several calls,
    asked again where the machine was busy."""
    for _ in range(4):
        a, b = _best_s(auto, reps), _best_s(pinned, reps)
        if a <= 1.5 * b + 40e-6:
            return
    pytest.fail(f"{a * 1e6:.0f} us against {b * 1e6:.0f} us")


@pytest.mark.parametrize("n,dim,max_h", [(400_000, 2, 4), (400_000, 8, 4), (200_000, 5, 1), (400_000, 3, 6)])
def test_few_dimensional_counts(n, dim, max_h):
    rows = G.gmm_rows(n, dim, 64, 0.2, seed=dim)
    with gts.Index(rows, 2, max_h=max_h) as a, gts.Index(rows, 2, max_h=max_h) as b:
        b.set_plain_threads(1, 256)
        for frac in (1e-4, 0.1):
            r = float(np.float32(G.quantile_radius(2, frac, 20000, 3, rows=rows)))
            for nq in (1, 8, 100, 443, 445, 1183, 1185, 2000):   # 296 CTAs are resident on a B200
                q = G.query_ids(n, nq, nq)
                np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
                if nq <= 100:
                    _not_slower(lambda: a.range(q, r), lambda: b.range(q, r))


@pytest.mark.parametrize("n,max_h", [(200_000, 2), (40_000, 1)])   # leaves of 20,000 and 40,000 words
def test_words_in_large_leaves(n, max_h):
    strs, lens = G.word_strings(n, 7)
    with gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h) as a, \
            gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h) as b:
        for mode in (0, 1):
            b.set_plain_threads(mode, 256)
        for nq in (8, 100):
            q = G.query_ids(n, nq, nq)
            for r in (1.0, 3.0):
                np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
                _not_slower(lambda: a.range(q, r), lambda: b.range(q, r))
            for x, y in zip(a.knn(q, 8, return_ids=True), b.knn(q, 8, return_ids=True)):
                np.testing.assert_array_equal(x, y)
            _not_slower(lambda: a.knn(q, 8), lambda: b.knn(q, 8))


@pytest.mark.parametrize("metric,n,dim,nq", [
    (1, 1000, 1000, 100), (0, 1000, 300, 60), (2, 1000, 300, 100), (5, 1000, 300, 100), (1, 2000, 33, 100),
    (1, 1000, 1000, 20), (2, 8000, 9, 100), (1, 5000, 64, 100), (5, 4000, 64, 40), (2, 2100, 128, 30)])
def test_small_indexes(metric, n, dim, nq):
    rows = G.gmm_rows(n, dim, 16, 0.3, seed=n + dim) + np.float32(0.5)
    q = G.query_ids(n, nq, nq)
    with gts.Index(rows, metric, max_h=3) as a, gts.Index(rows, metric, max_h=3) as b:
        for mode in (0, 1, 2):
            b.set_plain_threads(mode, 256)
        for k in (1, 16):
            for x, y in zip(a.knn(q, k, return_ids=True), b.knn(q, k, return_ids=True)):
                np.testing.assert_array_equal(x, y)
            _not_slower(lambda: a.knn(q, k), lambda: b.knn(q, k))
        r = float(np.median(a.knn(q, 16)))
        np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
        for x, y in zip(a.range_ids(q, r), b.range_ids(q, r)):
            np.testing.assert_array_equal(x, y)
        _not_slower(lambda: a.range(q, r), lambda: b.range(q, r))


@pytest.mark.parametrize("n,dim", [(1_000_000, 9), (1_000_000, 16), (500_000, 64)])
def test_selective_counts(n, dim):
    """Radii of no, few and many hits; the batch is asked from 1,024 queries on."""
    rng = np.random.default_rng(dim)
    rows = rng.standard_normal((n, dim), dtype=np.float32) * np.float32(0.15)
    rows += (rng.random((1024, dim), dtype=np.float32) * 4)[rng.integers(0, 1024, n)]
    rows[:500] = rows[500:1000]
    with gts.Index(rows, 2, max_h=6) as a, gts.Index(rows, 2, max_h=6) as b:
        b.set_plain_threads(1, 256)
        near = float(np.median(a.knn(G.query_ids(n, 64, 1), 2)))
        for nq in (33, 1023, 1024, 6000):
            q = np.concatenate([np.arange(20), G.query_ids(n, nq - 20, nq)]).astype(np.int32)
            for r in (0.0, 1e-3, near / 4, near, 1.5 * near):
                np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
                if nq >= 1024:
                    _not_slower(lambda: a.range(q, r), lambda: b.range(q, r), 3)


@pytest.mark.parametrize("n,max_h,lo,hi", [(8000, 2, 3, 16), (32768, 5, 3, 16), (30000, 4, 20, 50), (20000, 4, 70, 108)])
def test_words_few_short_and_long(n, max_h, lo, hi):
    """Small word lists, radii far below the lengths, strings past the sweep's words."""
    rng = np.random.default_rng(n)
    lens = rng.integers(lo, hi + 1, n).astype(np.int32)
    strs = np.where(np.arange(109)[None, :] < lens[:, None], rng.integers(97, 107, (n, 109)), 0).astype(np.uint8)
    with gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h) as a, \
            gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h) as b:
        for mode in (0, 1):
            b.set_plain_threads(mode, 256)
        for nq in (4, 100, 600):
            q = G.query_ids(n, nq, nq)
            for r in (0.0, 1.0, 8.0):
                np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
                _not_slower(lambda: a.range(q, r), lambda: b.range(q, r), 3)
        for x, y in zip(a.knn(q[:100], 8, return_ids=True), b.knn(q[:100], 8, return_ids=True)):
            np.testing.assert_array_equal(x, y)
        _not_slower(lambda: a.knn(q[:100], 8), lambda: b.knn(q[:100], 8), 3)


def _swept(idx, call):
    call()
    return idx.search_stats()["pivots"] == 0   # the sweep counts none


def test_large_batches_of_the_sweep_tune_nothing():
    rows = G.gmm_rows(20000, 24, 16, 0.3, seed=9)
    q = G.query_ids(20000, 8000, 10)
    with gts.Index(rows, 2, max_h=4) as idx:
        assert _swept(idx, lambda: idx.knn(q, 8))
        assert idx.plain_threads(0) == 256           # the traversal's default
        want = idx.knn(q[:100], 129, return_ids=True)
        n0 = idx.kernel_launches()
        first = idx.knn(q, 129, return_ids=True)     # past the sweep's k: the traversal's, and tuned now
        n1 = idx.kernel_launches()
        again = idx.knn(q, 129, return_ids=True)
        assert n1 - n0 > idx.kernel_launches() - n1
        assert idx.plain_threads(0) in (128, 256, 512)
        for x, y, z in zip(first, again, want):
            np.testing.assert_array_equal(x, y)
            np.testing.assert_array_equal(x[:100], z)


def test_a_pin_ends_with_the_index_or_the_default():
    n = 12000
    rows = G.gmm_rows(n, 24, 16, 0.3, seed=11)
    q = G.query_ids(n, 700, 12)
    r = float(np.float32(G.quantile_radius(2, 0.02, 20000, 13, rows=rows)))
    flags, ids = G.update_stream(n, 400, 14, max_in_size=10)
    with gts.Index(rows, 2, max_h=4) as idx:
        assert _swept(idx, lambda: idx.range(q, r))
        for mode in (0, 1):
            idx.set_plain_threads(mode, 128)
        assert not _swept(idx, lambda: idx.range(q, r)) and not _swept(idx, lambda: idx.knn(q, 8))
        idx.update_run(flags, ids, r)                 # rebuilds: a new tree, untuned
        assert idx.plain_threads(0) == 0 and idx.plain_threads(1) == 0
        q2 = (q % idx.info["num"]).astype(np.int32)
        assert _swept(idx, lambda: idx.range(q2, r)) and _swept(idx, lambda: idx.knn(q2, 8))
        idx.plain_split(64)
        assert not _swept(idx, lambda: idx.range(q2, r))
        idx.plain_split(32768)                        # the default
        assert _swept(idx, lambda: idx.range(q2, r))
