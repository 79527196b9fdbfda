"""Double-precision POTRF / POSV in 64-bit fixed point (orders from 17 on, above 32
with the workspace the wsqueries request): the edges of its 8-column blocks,
row groups and teams, and the data it hands back to the FP64 path.

Bar of the factor: |A - L L^T|_ij <= (n + 8) 2^-53 sqrt(a_ii a_jj). Every entry of
L is within 2^-60 of its row's scale 2^E_i <= 4 sqrt(a_ii) times the rounding of
its column's reciprocal root (below 2^-57) and is then rounded to FP64 (2^-53 of
itself), so the two factors of an entry lose at most about 2 (2^-53 + 2^-57) of
sqrt(a_ii a_jj) by Cauchy-Schwarz; a sum of K products loses at most 4 K 2^-60 of
16 sqrt(a_ii a_jj), below K 2^-53; the check's own FP64 product loses K 2^-53 more,
hence the n."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev
from test_gpu_chol import check_untouched, make_batch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def potrf(gpu, handle, kb, a, n, lda, array=False):
    batch = a.shape[0]
    fn = "kblas_potrf_batch_wsquery" if array else "kblas_potrf_batch_strided_wsquery"
    getattr(kb.lib(), fn)(handle.ptr, n, batch)
    assert handle.allocate_workspace() == 1
    da = to_dev(gpu, a)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    if array:
        pa = ptr_array(gpu, da)
        assert handle.call("kblasDpotrf_batch", "L", n, pa.data_ptr(), lda, batch, info.data_ptr()) == 1
    else:
        assert handle.call("kblasDpotrf_batch_strided", "L", n, da.data_ptr(), lda, n * lda, batch,
                           info.data_ptr()) == 1
    gpu.cuda.synchronize()
    assert handle.device_status() == 1
    return da.cpu().numpy(), info.cpu().numpy()


def check_factor(a, out, n, b):
    A = np.tril(a[b, :n, :n].T)
    A = A + np.tril(A, -1).T
    L = np.tril(out[b, :n, :n].T)
    d = np.sqrt(np.diag(A))
    r = np.abs((A - L @ L.T) / d[:, None] / d[None, :])
    assert r.max() <= (n + 8) * U, (b, r.max() / U)


@pytest.mark.parametrize("n", [17, 31, 32, 33, 39, 40, 41, 63, 65, 95, 97, 128, 130, 177, 193, 216, 225, 300])
@pytest.mark.parametrize("array", [False, True])
def test_block_edges(gpu, handle, kb, wl, n, array):
    lda = n + (1 if array else 0)
    a = make_batch(wl, 19, n, lda, np.float64, seed=n)
    out, info = potrf(gpu, handle, kb, a, n, lda, array)
    assert (info == 0).all()
    check_untouched(a, out, n)
    for b in range(19):
        check_factor(a, out, n, b)


@pytest.mark.parametrize("n", [105, 128, 217, 319, 320, 321])
def test_block_edges_many_systems(gpu, handle, kb, wl, n):
    """More than two systems per SM: one or two warps a system, the factor in L2."""
    few = make_batch(wl, 5, n, n, np.float64, seed=n)
    a = np.ascontiguousarray(np.tile(few, (70, 1, 1)))
    out, info = potrf(gpu, handle, kb, a, n, n)
    assert (info == 0).all()
    check_untouched(few, out[-5:], n)
    for b in range(5):
        check_factor(few, out, n, b)
    assert np.array_equal(out, np.tile(out[:5], (70, 1, 1)))


@pytest.mark.parametrize("data", ["cond", "cov", "graded", "huge", "tiny", "small_pivot"])
@pytest.mark.parametrize("n", [24, 48, 131])
def test_hard_data(gpu, handle, kb, wl, data, n):
    """graded rows keep to the fixed-point path; huge and tiny diagonals (beyond
    2^+-800) and pivots below 2^-42 take the FP64 path."""
    batch = 6
    rng = np.random.default_rng(n)
    if data == "cond":
        a = wl.spd_cond(batch, n, seed=n, logc=(2.0, 8.0))[0]
    elif data == "cov":
        a = wl.sqexp_cov(batch, n, seed=n)
    else:
        a = wl.spd_shifted(batch, n, seed=n)
    if data == "graded":
        d = 2.0 ** rng.integers(-300, 300, n)
        a = a * d[None, :, None] * d[None, None, :]
    elif data == "huge":
        a = a * 2.0 ** 850
    elif data == "tiny":
        a = a * 2.0 ** -850
    elif data == "small_pivot":
        k = n - 5
        for s in range(batch):
            L = np.linalg.cholesky(a[s])
            L[k, k] = 2.0 ** -22 * np.linalg.norm(L[k])
            a[s] = L @ L.T
    a = np.ascontiguousarray(a)
    out, info = potrf(gpu, handle, kb, a, n, n)
    assert (info == 0).all()
    for b in range(batch):
        check_factor(a, out, n, b)


@pytest.mark.parametrize("n", [20, 40, 70, 150])
@pytest.mark.parametrize("data", ["late", "large_row", "nan", "inf", "zero_pivot"])
def test_failures(gpu, handle, kb, wl, orc, n, data):
    """info is the oracle's, and A is left as it was from the failing column on
    (what the columns before it hold below the failing block is not defined)."""
    batch = 5
    a = make_batch(wl, batch, n, n, np.float64, seed=n + 1)
    r = n - 7
    for s in range(0, batch, 2):  # the others stay positive definite
        if data == "late":
            a[s, r, r] = -1.0
        elif data == "large_row":  # row r of L exceeds sqrt(a_rr) long before its pivot
            a[s, 2, r] = 50.0 * n
            a[s, 9, r] = -80.0 * n
        elif data == "nan":
            a[s, 5, r] = np.nan
        elif data == "inf":
            a[s, 5, r] = np.inf
        else:
            a[s, r, r] = 0.0
    ref = a.copy()
    info_ref = orc.potrf_batch(ref, n)
    out, info = potrf(gpu, handle, kb, a, n, n)
    assert np.array_equal(info, info_ref)
    assert (info[::2] > 0).all() and (info[1::2] == 0).all()
    check_untouched(a, out, n)
    for s in range(batch):
        if info[s] == 0:
            check_factor(a, out, n, s)
            continue
        k = info[s] - 1
        assert np.array_equal(out[s, k:], a[s, k:], equal_nan=True)


@pytest.mark.parametrize("n", [33, 64, 65, 100, 257, 300])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 9])
def test_solve_groups(gpu, handle, kb, wl, orc, n, m):
    """One and four right-hand sides to a warp, and segments of 64 / 256 rows."""
    batch, ldb = 7, m + 2
    a = make_batch(wl, batch, n, n, np.float64, seed=n + m)
    b = wl.rhs_rows(batch, m, n, seed=m, ld=ldb)
    kb.lib().kblas_posv_batch_strided_wsquery(handle.ptr, b"R", m, n, batch)
    assert handle.allocate_workspace() == 1
    da, db = to_dev(gpu, a), to_dev(gpu, b)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    assert handle.call("kblasDposv_batch_strided", "R", "L", m, n, da.data_ptr(), n, n * n,
                       db.data_ptr(), ldb, n * ldb, batch, info.data_ptr()) == 1
    gpu.cuda.synchronize()
    X = db.cpu().numpy()
    assert (info.cpu().numpy() == 0).all()
    eta = orc.backward_error_r(a, X, b, m, n)
    assert eta.max() <= 10 * n * U
    assert np.array_equal(X[:, :, m:], b[:, :, m:])
