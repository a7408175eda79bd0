"""The fast form's configurations as the ABI reports and takes them: every one
that can be chosen can be read, written back and read again, and answers as the
others do."""
import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu

KEYS = ("learned_seed", "col_groups", "item_blocks", "streamed", "by_block", "keeps_start")


def _write(idx, k, c):
    idx.set_fast_config(k, c["learned_seed"], c["col_groups"], c["item_blocks"], c["streamed"], c["by_block"],
                        c["keeps_start"])


@pytest.mark.parametrize("n,dim", [(12000, 64), (12000, 128), (9000, 200)])
def test_a_tuned_configuration_can_be_written_back(oracle, n, dim):
    rows = G.gmm_rows(n, dim, 24, 0.25, seed=dim)
    ds = oracle.Dataset(2, rows)
    q = G.query_ids(n, 2200, seed=22)
    with gts.Index(rows, 2, max_h=4) as idx, gts.Index(rows, 2, max_h=4) as other:
        for k in (1, 8, 64):
            want = idx.knn(q, k, form=gts.FORM_FAST, return_ids=True)
            tuned = idx.fast_config(k)
            assert tuned["tuned"]
            _write(other, k, tuned)
            assert {x: other.fast_config(k)[x] for x in KEYS} == {x: tuned[x] for x in KEYS}
            for x, y in zip(other.knn(q, k, form=gts.FORM_FAST, return_ids=True), want):
                np.testing.assert_array_equal(x, y)
            for x, y in zip(want, oracle.knn_brute(ds, q[:60], k)):
                np.testing.assert_array_equal(x[:60], y)


@pytest.mark.parametrize("streamed", [False, True])
@pytest.mark.parametrize("k", [1, 16, 33, 64])
def test_keeping_the_start_answers_as_the_heaps(oracle, k, streamed):
    rows = np.concatenate([G.gmm_rows(9000, 96, 24, 0.25, seed=3), np.tile(G.gmm_rows(2, 96, 1, 0.2, 4), (800, 1))])
    q = np.concatenate([G.query_ids(9000, 300, seed=5), [9000, 9001, 10599]]).astype(np.int32)   # the last ones overflow
    with gts.Index(rows, 2, max_h=4) as idx:
        idx.set_fast_config(k, False, 4, 8, streamed=streamed, keeps_start=True)
        c = idx.fast_config(k)
        assert c["keeps_start"] and c["streamed"] == streamed and c["col_groups"] == 4
        for x, y in zip(idx.knn(q, k, form=gts.FORM_FAST, return_ids=True), oracle.knn_brute(oracle.Dataset(2, rows), q, k)):
            np.testing.assert_array_equal(x, y)
        with pytest.raises(gts.GtsError):
            idx.set_fast_config(k, False, 2, 8, keeps_start=True)


@pytest.mark.parametrize("nq", [1, 64, 65])
def test_timing_does_not_change_what_runs(nq):
    rows = G.gmm_rows(9000, 64, 8, 0.3, seed=7)
    q = G.query_ids(9000, nq, 8)
    with gts.Index(rows, 2, max_h=4) as idx:
        idx.fast_graphs(False)
        counts = []
        for timed in (False, True):
            if timed:
                idx.filter_timing(reset=True)
            idx.knn(q, 8, form=gts.FORM_FAST)
            n0 = idx.kernel_launches()
            kth = idx.knn(q, 8, form=gts.FORM_FAST)
            counts.append((idx.kernel_launches() - n0, kth))
        ms, launches = idx.filter_timing()
        assert counts[0][0] == counts[1][0] and launches == 2 and 0 < ms < 1000
        np.testing.assert_array_equal(counts[0][1], counts[1][1])


@pytest.mark.parametrize("dim,nq,tiles", [(300, 51, False), (300, 52, True), (128, 64, False), (128, 65, True), (64, 64, False)])
def test_small_batches_by_width(oracle, dim, nq, tiles):
    rows = G.gmm_rows(6000, dim, 8, 0.3, seed=dim)
    q = G.query_ids(6000, nq, 9)
    with gts.Index(rows, 2, max_h=4) as idx:
        idx.prepare()
        n0 = idx.kernel_launches()
        got = idx.knn(q, 8, form=gts.FORM_FAST, return_ids=True)
        assert (idx.kernel_launches() - n0 > 3) == tiles
        for x, y in zip(got, oracle.knn_brute(oracle.Dataset(2, rows), q, 8)):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("dim", [130, 192, 250, 64])
def test_tuning_ends(oracle, dim):
    """The runs are bounded, also where the recheck that is tried last is the
    slower one."""
    rows = G.gmm_rows(6000, dim, 1, 1.0, seed=dim)
    q = G.query_ids(6000, 2100, 9)
    with gts.Index(rows, 2, max_h=3) as idx:
        idx.prepare()
        for k in (1, 8):
            n0 = idx.kernel_launches()
            got = idx.knn(q, k, form=gts.FORM_FAST, return_ids=True)
            assert idx.fast_config(k)["tuned"] and idx.kernel_launches() - n0 < 60 * 30   # 60 configurations at most
            for x, y in zip(got, oracle.knn_brute(oracle.Dataset(2, rows), q[:50], k)):
                np.testing.assert_array_equal(x[:50], y)
