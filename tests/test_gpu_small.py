"""The fast form's small batches (no tiles) against the tile path (a pinned
configuration) and brute force: batch sizes around its groups of eight and its
limit, widths of each kernel variant, k past the nearest blocks' objects, equal
objects that overflow its lists, a tuned large batch's few re-answered queries."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,comps,sigma,max_h", [
    (20000, 64, 16, 0.3, 5), (20000, 65, 16, 0.3, 5), (12000, 128, 1, 1.0, 4), (9000, 320, 8, 0.3, 4), (90, 16, 1, 1.0, 3),
    (1, 3, 1, 1.0, 2)])
def test_small_batches_equal_tiles_and_brute_force(oracle, n, dim, comps, sigma, max_h):
    rows = G.gmm_rows(n, dim, comps, sigma, seed=n + dim)
    ds = oracle.Dataset(2, rows)
    with gts.Index(rows, 2, max_h=max_h) as a, gts.Index(rows, 2, max_h=max_h) as b:
        for k in (1, 8, 33, 64):
            b.set_fast_config(k, False, 1)
            for nq in (1, 7, 8, 9, 64, 65):
                q = (np.arange(nq) * 37 % n).astype(np.int32)
                got = a.knn(q, k, form=gts.FORM_FAST, return_ids=True)
                for x, y, z in zip(got, b.knn(q, k, form=gts.FORM_FAST, return_ids=True), oracle.knn_brute(ds, q, k)):
                    np.testing.assert_array_equal(x, y, err_msg=f"k={k} nq={nq}")
                    np.testing.assert_array_equal(x, z, err_msg=f"k={k} nq={nq}")
                np.testing.assert_array_equal(a.knn(q, k, form=gts.FORM_FAST), got[0])


def test_full_lists_go_to_the_tiles(oracle):
    rows = np.concatenate([np.tile(G.gmm_rows(2, 32, 1, 0.1, 1), (1500, 1)), G.gmm_rows(9000, 32, 8, 0.3, 2)])
    q = np.array([0, 1, 5000, 2999, 11000], np.int32)
    with gts.Index(rows, 2, max_h=4) as idx:
        for x, y in zip(idx.knn(q, 8, form=gts.FORM_FAST, return_ids=True),
                        oracle.knn_brute(oracle.Dataset(2, rows), q, 8)):
            np.testing.assert_array_equal(x, y)
        many = np.concatenate([q, 3000 + G.query_ids(9000, 3000, 3)]).astype(np.int32)   # a few overflow among many
        np.testing.assert_array_equal(idx.knn(many, 8, form=gts.FORM_FAST)[:5],
                                      oracle.knn_brute(oracle.Dataset(2, rows), q, 8)[0])
