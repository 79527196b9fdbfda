"""Single-precision POTRF / POSV / POTRS on the one-row-per-lane kernel (orders 33
to about 330): the orders where its rows per lane, warps per system and place
change, and failing pivots in every position of its 8-column blocks. Bars of
test_gpu_chol.py: info exact, backward errors <= 10 n eps."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev
from test_gpu_chol import check_untouched, make_batch

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24


@pytest.mark.parametrize("n", [33, 63, 64, 65, 127, 128, 129, 247, 248, 249, 319, 332, 345])
@pytest.mark.parametrize("form", ["strided", "array"])
def test_posv_edges(gpu, handle, wl, orc, n, form):
    m, batch = 5, 11
    lda, ldb = n + 1, m + 2
    a = make_batch(wl, batch, n, lda, np.float32, seed=n)
    b = wl.rhs_rows(batch, m, n, seed=n, ld=ldb, dtype=np.float32)
    bad = [2, 7]
    for s in bad:
        c = n - 1 - 3 * s
        a[s, c, c] = -1.0
    da, db = to_dev(gpu, a), to_dev(gpu, b)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    if form == "strided":
        st = handle.call("kblasSposv_batch_strided", "R", "L", m, n, da.data_ptr(), lda, n * lda,
                         db.data_ptr(), ldb, n * ldb, batch, info.data_ptr())
    else:
        pa, pb = ptr_array(gpu, da), ptr_array(gpu, db)
        st = handle.call("kblasSposv_batch", "R", "L", m, n, pa.data_ptr(), lda, pb.data_ptr(), ldb,
                         batch, info.data_ptr())
    assert st == 1
    gpu.cuda.synchronize()
    ref = a.copy()
    info_ref = orc.potrf_batch(ref, n)
    assert np.array_equal(info.cpu().numpy(), info_ref)
    ok = info_ref == 0
    assert not ok[bad].any() and ok.sum() == batch - len(bad)
    X = db.cpu().numpy()
    eta = orc.backward_error_r(a[ok], X[ok], b[ok], m, n)
    assert eta.max() <= 10 * n * U32
    assert np.array_equal(X[~ok], b[~ok]) and np.array_equal(X[:, :, m:], b[:, :, m:])
    L = da.cpu().numpy()
    check_untouched(a, L, n)
    for s in np.flatnonzero(ok):
        assert orc.factor_backward_error(a[s], L[s], n) <= 10 * n * U32
    # the factor, solved with again
    db2 = to_dev(gpu, b)
    assert handle.call("kblasSpotrs_batch_strided", "R", "L", m, n, da.data_ptr(), lda, n * lda,
                       db2.data_ptr(), ldb, n * ldb, batch) == 1
    gpu.cuda.synchronize()
    eta = orc.backward_error_r(a[ok], db2.cpu().numpy()[ok], b[ok], m, n)
    assert eta.max() <= 10 * n * U32


@pytest.mark.parametrize("n", [33, 70, 150])
def test_failing_pivots(gpu, handle, wl, orc, n):
    """One system per failing column; NaN instead of a negative pivot in the odd ones."""
    a = make_batch(wl, n, n, n, np.float32, seed=3 * n)
    for s in range(n):
        a[s, s, s] = np.nan if s & 1 else -2.0
    da = to_dev(gpu, a)
    info = gpu.full((n,), -99, dtype=gpu.int32, device="cuda")
    assert handle.call("kblasSpotrf_batch_strided", "L", n, da.data_ptr(), n, n * n, n,
                       info.data_ptr()) == 1
    gpu.cuda.synchronize()
    assert np.array_equal(info.cpu().numpy(), np.arange(1, n + 1))
    check_untouched(a, da.cpu().numpy(), n)
