"""Range counts of few-dimensional rows (a query per warp) against the per-CTA
traversal (pinned threads) and brute force: every width and metric it takes,
tree orders up to its limit, radii from zero to everything (deep stacks), rows
given as data, handed-over items and the stream update's counts."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,dim,n,order,max_h,max_size", [
    (1, 2, 60000, 10, 5, 20), (2, 1, 30001, 10, 5, 20), (0, 3, 20000, 16, 4, 20), (2, 8, 20000, 2, 14, 3),
    (1, 7, 9000, 3, 8, 1), (2, 4, 500, 10, 1, 20), (1, 5, 3000, 16, 3, 5), (2, 2, 40000, 10, 2, 20),
    (2, 2, 20000, 17, 4, 20),   # an order it leaves to the CTA traversal
])
def test_warp_range_counts(oracle, metric, dim, n, order, max_h, max_size):
    rows = G.hotspot_points(n, 5) if dim == 2 else G.gmm_rows(n, dim, 20, 0.2, seed=n)
    rows[10:30] = rows[100:120]
    ds = oracle.Dataset(metric, rows)
    q = np.concatenate([np.arange(10, 30), G.query_ids(n, min(n, 700), 6)]).astype(np.int32)
    new = rows[q[:100]] + np.float32(1e-3)
    kw = dict(tree_order=order, max_h=max_h, max_size=max_size)
    with gts.Index(rows, metric, **kw) as a, gts.Index(rows, metric, **kw) as b:
        b.set_plain_threads(1, 256)
        radii = [0.0, 1e30] + [float(np.float32(G.quantile_radius(metric, f, 20000, 7, rows=rows))) for f in (1e-3, 0.3)]
        radii.append(float(np.float32(radii[-1] * 50)))
        for r in radii:
            got = a.range(q, r)
            np.testing.assert_array_equal(got, b.range(q, r), err_msg=f"r={r}")
            np.testing.assert_array_equal(got[:100], oracle.range_brute(ds, q[:100], r), err_msg=f"r={r}")
            np.testing.assert_array_equal(a.range_rows(new, r), b.range_rows(new, r), err_msg=f"r={r}")
        before = a.plain_split(16)
        np.testing.assert_array_equal(a.range(q, radii[-1]), b.range(q, radii[-1]))
        if order <= 16 and n >= 20000 and max_h > 3:
            assert a.plain_split() > before   # items were handed over
        flags, ids = G.update_stream(n, 600, 8)
        np.testing.assert_array_equal(a.update_run(flags, ids, radii[2])[0], b.update_run(flags, ids, radii[2])[0])
