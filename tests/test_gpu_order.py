"""The block order's assignment kernel where its tiles and dimensions end: the
fast form answers what brute force does over blocks ordered by it (segments
split by k-means, halved, at the edge of a block), aligned and unaligned rows,
and every object has exactly one slot."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,comps,sigma", [
    (128, 16, 1, 1.0), (129, 17, 1, 1.0), (257, 4, 2, 0.1), (1025, 1, 4, 0.2), (5000, 15, 8, 0.2), (5000, 128, 8, 0.2),
    (20011, 129, 24, 0.3), (9000, 320, 4, 0.3), (9000, 318, 4, 0.3)])
def test_blocks_hold_every_object_once(oracle, n, dim, comps, sigma):
    rows = G.gmm_rows(n, dim, comps, sigma, seed=n + dim)
    rows[n // 2:n // 2 + min(200, n // 4)] = rows[0]   # equal objects: a segment k-means cannot split
    q = (np.arange(300) * 41 % n).astype(np.int32)
    with gts.Index(rows, 2, max_h=3) as idx:
        got = idx.knn(q, 4, form=gts.FORM_FAST, return_ids=True)
        for x, y in zip(got, oracle.knn_brute(oracle.Dataset(2, rows), q, 4)):
            np.testing.assert_array_equal(x, y)
        # a radius over everything counts each object once
        np.testing.assert_array_equal(idx.range(q[:9], 1e6, form=gts.FORM_FAST), np.full(9, n))
