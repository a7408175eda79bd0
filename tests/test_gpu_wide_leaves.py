"""kNN by the traversal over leaves of hundreds and thousands of objects, where a
step verifies as many as fit: few-dimensional rows, wide trees, k past the
sweep's, strings; the same answers from every call."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,n,dim,order,max_h,max_size,k", [
    (1, 60000, 3, 30, 3, 50, 8), (2, 50000, 2, 10, 2, 20, 8), (0, 30000, 8, 10, 1, 20, 1), (2, 40000, 5, 16, 3, 20, 128),
    (2, 30000, 24, 10, 2, 20, 200), (1, 20000, 40, 20, 2, 20, 256), (2, 60000, 1, 10, 3, 20, 33)])
def test_rows(oracle, metric, n, dim, order, max_h, max_size, k):
    rows = G.gmm_rows(n, dim, 40, 0.3, seed=n + dim)
    ds = oracle.Dataset(metric, rows)
    q = G.query_ids(n, 60, 5)
    want = oracle.knn_brute(ds, q, k)
    with gts.Index(rows, metric, tree_order=order, max_h=max_h, max_size=max_size) as idx:
        for nt in (0, 128, 256, 512):
            idx.set_plain_threads(0, nt)
            for _ in range(3):
                for x, y in zip(idx.knn(q, k, return_ids=True), want):
                    np.testing.assert_array_equal(x, y)


def test_strings(oracle):
    strs, lens = G.word_strings(30000, 9)
    ds = oracle.Dataset(6, strs=strs, lens=lens)
    q = G.query_ids(30000, 40, 5)
    with gts.Index(None, 6, strs=strs, lens=lens, max_h=2) as idx:
        for k in (20, 200):
            want = oracle.knn_brute(ds, q, k)
            idx.set_plain_threads(0, 256)
            for x, y in zip(idx.knn(q, k, return_ids=True), want):
                np.testing.assert_array_equal(x, y)
