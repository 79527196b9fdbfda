"""Double-precision POTRF / POSV of orders 17..32 on both sides of one wave of warps
(16 per SM): below it matrices that do not fit fixed point are factored again by the same
warp, above it (order 25 on) by a second launch that finds them by their mark in info, and
orders up to 24 or calls without info run on teams of lanes. Bars of test_gpu_chol.py."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev
from test_gpu_chol import check_untouched, make_batch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def mixed_batch(wl, n, lda):
    """12 systems: fitting ones, and every reason to leave fixed point."""
    a = make_batch(wl, 12, n, lda, np.float64, seed=n)
    low = np.tril(np.ones((n, n), bool), -1).T
    a[1, :, :n][low] *= 1e-9                      # weak couplings
    a[3, n - 2, n - 2] = -1.0                     # fails late
    a[4, 0, 0] = -1.0                             # fails at once
    a[6, 3, 7] = np.nan
    a[8, :, :n][np.tril(np.ones((n, n), bool)).T] *= 2.0 ** 850
    a[9, 5, 5] = 0.0
    a[10, 2, 9] = 40.0 * n                        # a row beyond its bound
    return a


@pytest.mark.parametrize("n", [17, 24, 25, 31, 32])
@pytest.mark.parametrize("copies", [20, 250])
@pytest.mark.parametrize("form,with_info", [("strided", True), ("array", True), ("strided", False)])
def test_posv(gpu, handle, wl, orc, n, copies, form, with_info):
    m, lda = 2, n + 1
    few = mixed_batch(wl, n, lda)
    bfew = wl.rhs_rows(12, m, n, seed=n, ld=m)
    ref = few.copy()
    info_ref = orc.potrf_batch(ref, n)
    assert (info_ref > 0).sum() == 5
    a, b = np.tile(few, (copies, 1, 1)), np.tile(bfew, (copies, 1, 1))
    batch = a.shape[0]
    da, db = to_dev(gpu, a), to_dev(gpu, b)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    pinfo = info.data_ptr() if with_info else 0
    if form == "strided":
        st = handle.call("kblasDposv_batch_strided", "R", "L", m, n, da.data_ptr(), lda, n * lda,
                         db.data_ptr(), m, n * m, batch, pinfo)
    else:
        pa, pb = ptr_array(gpu, da), ptr_array(gpu, db)
        st = handle.call("kblasDposv_batch", "R", "L", m, n, pa.data_ptr(), lda, pb.data_ptr(), m,
                         batch, pinfo)
    assert st == 1
    gpu.cuda.synchronize()
    if with_info:
        assert np.array_equal(info.cpu().numpy(), np.tile(info_ref, copies))
    L, X = da.cpu().numpy(), db.cpu().numpy()
    for c in (0, copies - 1):
        s = slice(12 * c, 12 * c + 12)
        check_untouched(few, L[s], n)
        ok = info_ref == 0
        assert np.array_equal(X[s][~ok], bfew[~ok])
        eta = orc.backward_error_r(few[ok], X[s][ok], bfew[ok], m, n)
        assert eta.max() <= 10 * n * U
        for q in np.flatnonzero(ok):
            assert orc.factor_backward_error(few[q], L[s][q], n) <= 10 * n * U
    assert np.array_equal(L, np.tile(L[:12], (copies, 1, 1)), equal_nan=True)
    assert np.array_equal(X, np.tile(X[:12], (copies, 1, 1)), equal_nan=True)
