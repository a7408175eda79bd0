"""The plain form's batched sweep against the per-query traversal (chosen by
pinning its threads) and the oracle's brute force: every metric it takes, row
widths around its 16-dimension stages and 4-float loads, batches around its
32- and 128-query tiles, lists that overflow (further rounds, the traversal),
long hit lists, duplicates, deep and shallow trees."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


def _pair(rows, metric, **kw):
    """An index that sweeps and one that traverses."""
    a, b = gts.Index(rows, metric, **kw), gts.Index(rows, metric, **kw)
    for mode in (0, 1, 2):
        b.set_plain_threads(mode, 256)
    return a, b


def _same(x, y):
    for u, v in zip(x, y):
        np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("metric,n,dim,comps,sigma,max_h,nq,k", [
    (2, 33000, 16, 40, 0.3, 5, 128, 8),      # one stage
    (2, 32801, 17, 40, 0.3, 5, 129, 1),      # a ragged second stage, 4-byte loads, a second tile
    (2, 40000, 300, 8, 1.0, 5, 33, 64),      # bounds that cut little
    (2, 33001, 128, 64, 0.2, 3, 1, 33),      # one query, leaves of hundreds
    (2, 33001, 9, 5, 0.3, 1, 32, 8),         # a root without children
    (1, 33003, 33, 40, 0.3, 5, 200, 16),
    (0, 33000, 12, 40, 0.3, 4, 140, 7),
    (5, 33005, 50, 40, 0.4, 5, 150, 10),
    (5, 33005, 64, 1, 0.05, 2, 5, 128),
    (2, 3000, 24, 10, 0.3, 4, 900, 5),       # a small index under a large batch
])
def test_sweep_equals_traversal_and_brute_force(oracle, metric, n, dim, comps, sigma, max_h, nq, k):
    rows = G.gmm_rows(n, dim, comps, sigma, seed=n + dim)
    if metric == 5:
        rows = rows + 0.5
    rows[5:40] = rows[1000:1035]   # equal objects
    q = np.concatenate([np.arange(5, min(nq, 20) + 5), G.query_ids(n, nq, seed=n)])[:nq].astype(np.int32)
    new = rows[q[:50]] + np.float32(0.01)
    a, b = _pair(rows, metric, max_h=max_h)
    with a, b:
        got = a.knn(q, k, return_ids=True)
        _same(got, b.knn(q, k, return_ids=True))
        _same(a.knn_rows(new, k, return_ids=True), b.knn_rows(new, k, return_ids=True))
        for frac in (0.0005, 0.02):
            r = float(np.float32(G.quantile_radius(metric, frac, 20000, 7, rows=rows)))
            counts = a.range(q, r)
            np.testing.assert_array_equal(counts, b.range(q, r))
            np.testing.assert_array_equal(a.range_rows(new, r), b.range_rows(new, r))
            hits = a.range_ids(q[:40], r)
            _same(hits, b.range_ids(q[:40], r))
            np.testing.assert_array_equal(hits[0], counts[:40])
        if metric != 5:   # the host's acosf may differ in the last bit
            bk, bi, bd = oracle.knn_brute(oracle.Dataset(metric, rows), q[:40], k)
            _same([x[:40] for x in got], (bk, bi, bd))


def _words(n, seed, long_ones):
    strs, lens = G.word_strings(n, seed)
    rng = np.random.default_rng(seed)
    for i, length in enumerate(long_ones):   # the pattern word and packed-text limits, and beyond
        strs[i] = 0
        strs[i, :length] = rng.integers(97, 123, length)
        lens[i] = length
    strs[60, :lens[60]] = 200                # bytes above 127
    lens[61:64] = 0                          # empty strings
    strs[61:64] = 0
    return strs, lens


@pytest.mark.parametrize("n,max_h,nq,k", [(20000, 4, 300, 16), (16501, 3, 1, 5), (40000, 5, 33, 128), (20000, 1, 31, 1)])
def test_string_sweep_equals_traversal_and_brute_force(oracle, n, max_h, nq, k):
    strs, lens = _words(n, n + 1, [31, 32, 33, 34, 63, 64, 65, 108])
    ds = oracle.Dataset(6, strs=strs, lens=lens)
    short = np.argsort(lens, kind="stable")[:20]   # heavy: thousands of close words
    q = np.concatenate([np.arange(8), [60, 61], short, G.query_ids(n, nq, 9)])[-max(nq, 1):].astype(np.int32) \
        if nq < 40 else np.concatenate([np.arange(8), [60, 61], short, G.query_ids(n, nq, 9)]).astype(np.int32)
    qs, ql = strs[q].copy(), lens[q].copy()
    qs[:, 0] = np.where(ql > 0, 113, qs[:, 0])     # new words: not in the index as such
    a = gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h)
    b = gts.Index(None, 6, strs=strs, lens=lens, max_h=max_h)
    for mode in (0, 1, 2):
        b.set_plain_threads(mode, 256)
    with a, b:
        got = a.knn(q, k, return_ids=True)
        _same(got, b.knn(q, k, return_ids=True))
        _same([x[:40] for x in got], oracle.knn_brute(ds, q[:40], k))
        _same(a.knn_rows((qs, ql), k, return_ids=True), b.knn_rows((qs, ql), k, return_ids=True))
        for r in (0.0, 1.0, 2.5, 3.0, 40.0):
            counts = a.range(q, r)
            np.testing.assert_array_equal(counts, b.range(q, r))
            np.testing.assert_array_equal(counts[:40], oracle.range_brute(ds, q[:40], r))
            np.testing.assert_array_equal(a.range_rows((qs, ql), r), b.range_rows((qs, ql), r))


def test_string_stream_counts():
    strs, lens = G.word_strings(20000, 31)
    flags, ids = G.update_stream(20000, 2000, 32, max_in_size=10)
    a = gts.Index(None, 6, strs=strs, lens=lens, max_h=4)
    b = gts.Index(None, 6, strs=strs, lens=lens, max_h=4)
    b.set_plain_threads(1, 256)
    with a, b:
        np.testing.assert_array_equal(a.update_run(flags, ids, 2.0)[0], b.update_run(flags, ids, 2.0)[0])


def test_overflowing_lists_and_long_hit_lists(oracle):
    """Thousands of equal distances overflow the candidate lists in every
    round; more hits than a list holds make range ids go over the rows again."""
    rows = np.concatenate([np.tile(G.gmm_rows(4, 20, 1, 0.1, 1), (3000, 1)), G.gmm_rows(25000, 20, 30, 0.3, 2)])
    q = np.concatenate([np.arange(0, 40), 12000 + G.query_ids(25000, 100, 3)]).astype(np.int32)
    ds = oracle.Dataset(2, rows)
    a, b = _pair(rows, 2, max_h=5)
    with a, b:
        got = a.knn(q, 9, return_ids=True)
        _same(got, b.knn(q, 9, return_ids=True))
        _same(got, oracle.knn_brute(ds, q, 9))
        for r in (0.0, 0.5):
            hits = a.range_ids(q, r)
            _same(hits, b.range_ids(q, r))
            np.testing.assert_array_equal(hits[0], oracle.range_brute(ds, q, r))
        assert hits[0].max() > 2048


def test_a_bad_device_id_is_reported():
    import torch
    rows = G.gmm_rows(33000, 24, 10, 0.3, 5)
    with gts.Index(rows, 2, max_h=5) as idx:
        want = idx.knn(np.arange(64, dtype=np.int32), 4)
        ids = torch.arange(64, dtype=torch.int32, device="cuda")
        ids[7] = 33000
        out = torch.zeros(64, dtype=torch.float32, device="cuda")
        with pytest.raises(gts.GtsError):
            idx.knn_device(ids.data_ptr(), 64, 4, out.data_ptr())
        got = out.cpu().numpy()
        assert np.isnan(got[7])
        np.testing.assert_array_equal(np.delete(got, 7), np.delete(want, 7))
