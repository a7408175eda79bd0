"""Seeds of objects whose block straddles two groups, and the filter that keeps
the bound a query starts with: a seed never lies below the k-th distance, the
few far ones are brought near it, the answers are brute force's."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,comps,sigma", [(60, 8, 2, 0.1), (1500, 16, 3, 0.05), (40000, 128, 37, 0.2),
                                               (30000, 300, 29, 0.2)])
def test_seeds_bound_and_answers(oracle, n, dim, comps, sigma):
    rows = G.gmm_rows(n, dim, comps, sigma, seed=n + dim)
    q = np.arange(0, n, max(1, n // 3000)).astype(np.int32)
    with gts.Index(rows, 2, max_h=3) as idx:
        for k in (8, 64):
            if k > n // 2:
                continue
            for _ in range(2):   # tuned on the first call, then the chosen filter
                got = idx.knn(q, k, form=gts.FORM_FAST, return_ids=True)
            want = oracle.knn_brute(oracle.Dataset(2, rows), q[:400], k)
            for x, y in zip(got, want):
                np.testing.assert_array_equal(x[:400], y)
            kth = got[0].astype(np.float64) ** 2
            seeds = idx.fast_seeds(q, k)
            assert (seeds >= kth * (1 - 1e-6)).all()
            if n >= 30000:   # 2.25 (the ratio that lists an object) and the widening
                assert np.percentile(seeds / np.median(kth), 99.9) < 2.5
