"""Single-precision POTRF of the orders that four warps share (129 to about 330):
every warp reads a block's 8 pivot rows from A, which the same call overwrites with
L. The call leaves the same bits in every copy of a matrix, in a batch that keeps
many CTAs on the GPU and in one that leaves it almost empty, and they are a factor
of the matrix (bar of test_gpu_chol.py: backward error <= 10 n eps). Failing pivots
leave the columns before them as the factor of the leading block and A's own entries
from the failing column on, in the pivot rows of the failing block too."""
import numpy as np
import pytest

from gpu_util import to_dev
from test_gpu_chol import check_untouched, make_batch

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24


def potrf(gpu, handle, a, n):
    lda, batch = a.shape[2], a.shape[0]
    da = to_dev(gpu, a)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    assert handle.call("kblasSpotrf_batch_strided", "L", n, da.data_ptr(), lda, n * lda, batch,
                       info.data_ptr()) == 1
    gpu.cuda.synchronize()
    return da.cpu().numpy(), info.cpu().numpy()


@pytest.mark.parametrize("n", [129, 136, 200, 249, 330])
def test_copies_agree(gpu, handle, wl, orc, n):
    few = make_batch(wl, 3, n, n + 1, np.float32, seed=n)
    alone, info = potrf(gpu, handle, few, n)
    assert (info == 0).all()
    check_untouched(few, alone, n)
    for s in range(3):
        assert orc.factor_backward_error(few[s], alone[s], n) <= 10 * n * U32
    many = np.ascontiguousarray(np.tile(few, (300, 1, 1)))
    for _ in range(3):
        out, info = potrf(gpu, handle, many, n)
        assert (info == 0).all()
        assert np.array_equal(out, np.tile(alone, (300, 1, 1)), equal_nan=True)


@pytest.mark.parametrize("n", [130, 260])
@pytest.mark.parametrize("at", [0, 1, 7, 8, 65, 128, -1])
def test_failing_block(gpu, handle, wl, orc, n, at):
    """The leading rows of a failing block hold L, as the same rows of a batch that
    does not fail do."""
    k = at % n
    good = make_batch(wl, 9, n, n, np.float32, seed=n + 3)
    full, info = potrf(gpu, handle, good, n)
    assert (info == 0).all()
    a = good.copy()
    a[:, k, k] = -1.0
    out, info = potrf(gpu, handle, a, n)
    assert np.array_equal(info, np.full(9, k + 1))
    check_untouched(a, out, n)
    low = np.tril(np.ones((n, n), bool)).T  # [column, row]
    for s in range(9):
        lead = low.copy()
        lead[k:, :] = lead[:, k:] = False
        assert np.array_equal(out[s][lead], full[s][lead])
        rest = low.copy()
        rest[:k, :] = False
        assert np.array_equal(out[s][rest], a[s][rest])
