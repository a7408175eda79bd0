"""Query ids given in device memory, some of them out of range: every form
leaves those queries out, marks their answers, answers the rest and reports an
error, whichever kernels it takes for the batch; the index answers the next
call as before."""
import ctypes as C

import numpy as np
import pytest

import gts_b200 as gts
from gts_b200 import datagen as G

pytestmark = pytest.mark.gpu

N, DIM = 20000, 48


@pytest.fixture(scope="module")
def index():
    with gts.Index(G.gmm_rows(N, DIM, 16, 0.3, 7), 2, max_h=4) as idx:
        idx.learn_radius(n_train=4000, k_max=8, epochs=2, seed=1)
        yield idx


def _ids(nq, bad):
    import torch
    q = G.query_ids(N, nq, nq)
    ids = q.copy()
    at = np.array([0, nq // 2, nq - 1][:len(bad)])
    ids[at] = bad
    return q, at, torch.from_numpy(ids).cuda()


# 5 and 64: without tiles; 65: one tile and a bit, no tuning; 600: several;
# 2,500: the tuner runs every filter variant on the batch
@pytest.mark.parametrize("nq", [5, 64, 65, 600, 2500])
@pytest.mark.parametrize("form", [gts.FORM_PLAIN, gts.FORM_FAST, gts.FORM_PLAIN_LEARNED])
def test_knn_ids_out_of_range(index, form, nq):
    import torch
    q, at, ids = _ids(nq, [N, -1, 2**31 - 1])
    want = index.knn(q, 8, form=form) if nq < 2048 else index.knn(q, 8)
    out = torch.zeros(nq, dtype=torch.float32, device="cuda")
    with pytest.raises(gts.GtsError, match="out of range"):
        index.knn_device(ids.data_ptr(), nq, 8, out.data_ptr(), form=form)
    got = out.cpu().numpy()
    assert np.isnan(got[at]).all()
    if form != gts.FORM_PLAIN_LEARNED:   # its queries of too small a radius are answered after the report
        np.testing.assert_array_equal(np.delete(got, at), np.delete(want, at))
    np.testing.assert_array_equal(index.knn(q, 8, form=form), want)


@pytest.mark.parametrize("nq", [5, 300, 2500])
@pytest.mark.parametrize("form", [gts.FORM_PLAIN, gts.FORM_FAST])
def test_range_ids_out_of_range(index, form, nq):
    import torch
    q, at, ids = _ids(nq, [N + 5, -7])
    r = float(np.median(index.knn(q[:64], 8)))
    want = index.range(q, r, form=form)
    out = torch.zeros(nq, dtype=torch.int32, device="cuda")
    with pytest.raises(gts.GtsError, match="out of range"):
        index.range_device(ids.data_ptr(), nq, r, out.data_ptr(), form=form)
    got = out.cpu().numpy()
    assert (got[at] == -1).all()
    np.testing.assert_array_equal(np.delete(got, at), np.delete(want, at))
    np.testing.assert_array_equal(index.range(q, r, form=form), want)


def test_fixed_scratch_ids_out_of_range(index):
    import torch
    q, at, ids = _ids(300, [N])
    want = index.knn(q, 8)
    index.prepare()
    out = torch.zeros(300, dtype=torch.float32, device="cuda")
    lib = gts._load_lib()
    rc = lib.gts_knn_device_noalloc(index._h, C.c_void_p(ids.data_ptr()), 300, 8, C.c_void_p(out.data_ptr()), None, None,
                                    None)
    assert rc == -5 and b"out of range" in lib.gts_last_error()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.isnan(got[at]).all()
    np.testing.assert_array_equal(np.delete(got, at), np.delete(want, at))
