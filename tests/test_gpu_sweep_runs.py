"""Batches that the sweep answers in several runs (more than 4,096 queries of
rows, 2,048 strings, or fewer where the budget gives it fewer tiles), compared
in full with the per-query traversal: every answer of every run, lists that
overflow in one run and not in the next, hit lists made longer on the way."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu

MB = 1 / 1024


def _swept(idx, call):
    out = call()
    assert idx.search_stats()["pivots"] == 0   # the sweep counts none
    return out


def _same(x, y):
    for u, v in zip(x, y):
        np.testing.assert_array_equal(u, v)


def _indexes(budget, *args, **kw):
    a, b = gts.Index(*args, mem_budget_gb=budget, **kw), gts.Index(*args, **kw)
    for mode in (0, 1, 2):
        b.set_plain_threads(mode, 256)
    return a, b


# 0: 32 tiles of 128 queries; 24 MiB: eight or so; 4 MiB: one
@pytest.mark.parametrize("metric,dim,nq,budget", [
    (2, 24, 5000, 0), (1, 33, 4097, 0), (5, 16, 4300, 0), (2, 100, 3000, 24 * MB), (2, 24, 700, 4 * MB), (0, 40, 900, 4 * MB)])
def test_rows_in_several_runs(metric, dim, nq, budget):
    n = 33000
    rows = G.gmm_rows(n, dim, 30, 0.3, seed=dim) + np.float32(0.5 if metric == 5 else 0)
    rows[20000:22500] = rows[19999]            # 2,501 equal objects: full lists
    q = G.query_ids(n, nq, nq)
    q[[3, nq - 2]] = [20000, 20001]            # in the first run and in the last
    new = rows[q] + np.float32(0.01)
    r = float(np.float32(G.quantile_radius(metric, 0.03, 20000, 7, rows=rows)))
    a, b = _indexes(budget, rows, metric, max_h=4)
    with a, b:
        for k in (1, 9):
            _same(a.knn(q, k, return_ids=True), b.knn(q, k, return_ids=True))
            _same(a.knn_rows(new, k, return_ids=True), b.knn_rows(new, k, return_ids=True))
        np.testing.assert_array_equal(_swept(a, lambda: a.range(q, r)), b.range(q, r))
        np.testing.assert_array_equal(_swept(a, lambda: a.range_rows(new, r)), b.range_rows(new, r))
        _same(a.range_ids(q, r / 2), b.range_ids(q, r / 2))
        clean = q[(q < 19999) | (q >= 22500)]
        a.knn(clean, 9)
        assert a.search_stats()["pivots"] < len(clean)   # the traversal answered few of them if any


@pytest.mark.parametrize("nq,budget", [(5000, 0), (600, 24 * MB)])
def test_hit_lists_grow_in_a_later_run(nq, budget):
    n = 33000
    rows = G.gmm_rows(n, 20, 30, 0.3, seed=2)
    rows[20000:23000] = rows[19999] + G.gmm_rows(3000, 20, 1, 0.001, seed=3) * np.float32(1e-3)
    a, b = _indexes(budget, rows, 2, max_h=5)
    with a, b:
        q = G.query_ids(19000, nq, nq)
        for at in (nq - 1, 0):                 # the long list in the last run, then in the first
            x = q.copy()
            x[at] = 20500
            got = a.range_ids(x, 0.3)
            assert got[0][at] > 2048
            _same(got, b.range_ids(x, 0.3))


@pytest.mark.parametrize("nq,budget", [(3000, 0), (2100, 40 * MB), (700, 5 * MB)])
def test_strings_in_several_runs(nq, budget):
    n = 40000
    strs, lens = G.word_strings(n, 11)
    rng = np.random.default_rng(12)
    for i, length in enumerate([31, 32, 33, 34, 63, 64, 65, 108]):
        strs[i] = 0
        strs[i, :length] = rng.integers(97, 123, length)
        lens[i] = length
    short = np.argsort(lens, kind="stable")[:30]   # thousands of close words
    q = np.concatenate([np.arange(8), short, G.query_ids(n, nq, 13)])[:nq].astype(np.int32)
    rng.shuffle(q)
    qs, ql = strs[q].copy(), lens[q].copy()
    qs[:, 0] = np.where(ql > 0, 113, qs[:, 0])
    a, b = _indexes(budget, None, 6, strs=strs, lens=lens, max_h=5)
    with a, b:
        for k in (1, 20):
            _same(a.knn(q, k, return_ids=True), b.knn(q, k, return_ids=True))
        _same(a.knn_rows((qs, ql), 8, return_ids=True), b.knn_rows((qs, ql), 8, return_ids=True))
        plain = np.array([i for i in q if lens[i] <= 32], np.int32)
        for r in (1.0, 2.0, 5.0):
            np.testing.assert_array_equal(a.range(q, r), b.range(q, r))
            np.testing.assert_array_equal(a.range_rows((qs, ql), r), b.range_rows((qs, ql), r))
            _swept(a, lambda: a.range(plain, r))


@pytest.mark.parametrize("lo,hi,max_h", [(1, 32, 5), (20, 50, 4), (40, 64, 5), (30, 70, 2)])
def test_long_strings(oracle, lo, hi, max_h):
    """Patterns on both sides of a 32-bit word, in one pass or two, few and many."""
    n = 34000
    rng = np.random.default_rng(lo)
    lens = rng.integers(lo, hi + 1, n).astype(np.int32)
    strs = np.where(np.arange(109)[None, :] < lens[:, None], rng.integers(97, 101, (n, 109)), 0).astype(np.uint8)
    strs[100:2400] = strs[99]                  # equal strings: full lists
    lens[100:2400] = lens[99]
    a, b = _indexes(0, None, 6, strs=strs, lens=lens, max_h=max_h)
    with a, b:
        for nq in (20, 600):
            q = np.concatenate([[99, 100], 2400 + G.query_ids(n - 2400, nq, nq)]).astype(np.int32)
            for k in (1, 12):
                got = a.knn(q, k, return_ids=True)
                _same(got, b.knn(q, k, return_ids=True))
            _same([x[:6] for x in got], oracle.knn_brute(oracle.Dataset(6, strs=strs, lens=lens), q[:6], 12))
            for r in (0.0, 3.0, 0.45 * hi):
                np.testing.assert_array_equal(a.range(q, r), b.range(q, r))


@pytest.mark.parametrize("budget", [0, 6 * MB])
def test_a_stream_in_several_runs(budget):
    n = 20000
    rows = G.gmm_rows(n, 24, 20, 0.3, seed=15)
    flags, ids = G.update_stream(n, 48000 if not budget else 12000, 16, max_in_size=10)
    assert (flags == 2).sum() > (4100 if not budget else 1000)
    r = float(np.float32(G.quantile_radius(2, 0.02, 20000, 17, rows=rows)))
    a, b = _indexes(budget, rows, 2, max_h=4)
    with a, b:
        np.testing.assert_array_equal(a.update_run(flags, ids, r)[0], b.update_run(flags, ids, r)[0])
