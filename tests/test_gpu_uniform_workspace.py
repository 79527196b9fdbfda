"""Uniform double-precision POTRF / POTRS / POSV above order 32: the workspace that a query
for a small batch requests serves a larger one on the same kernels (bit for bit the results
under the larger query), and batches of more systems than the list of those left to FP64
holds (65,536) run in slices."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev
from test_gpu_chol import make_batch

pytestmark = pytest.mark.gpu


def posv(gpu, h, kb, a, b, query_batch):
    batch, n, m = b.shape
    kb.lib().kblas_posv_batch_strided_wsquery(h.ptr, b"R", m, n, query_batch)
    assert h.allocate_workspace() == 1
    da, db = to_dev(gpu, a), to_dev(gpu, b)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    assert h.call("kblasDposv_batch_strided", "R", "L", m, n, da.data_ptr(), n, n * n, db.data_ptr(),
                  m, n * m, batch, info.data_ptr()) == 1
    gpu.cuda.synchronize()
    return da.cpu().numpy(), db.cpu().numpy(), info.cpu().numpy()


@pytest.mark.parametrize("n", [40, 110, 330])
def test_query_for_a_smaller_batch(gpu, kb, wl, n):
    few = make_batch(wl, 8, n, n, np.float64, seed=n)
    few[3, n - 2, n - 2] = -1.0
    a = np.ascontiguousarray(np.tile(few, (50, 1, 1)))
    b = wl.rhs_rows(400, 2, n, seed=n, ld=2)
    got = []
    for q in (1, 400):
        h = kb.Handle()
        got.append(posv(gpu, h, kb, a, b, q))
        h.close()
    assert (got[0][2] == np.tile([0, 0, 0, n - 1, 0, 0, 0, 0], 50)).all()
    for x, y in zip(*got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("form", ["strided", "array"])
def test_slices(gpu, handle, kb, wl, form):
    n, m, extra = 33, 1, 11
    batch = 65536 + extra
    few = make_batch(wl, 64, n, n, np.float64, seed=5)
    for s in (0, 5, 63):
        few[s, n - 1 - s % 7, n - 1 - s % 7] = -1.0
    want = np.zeros(64, np.int32)
    want[[0, 5, 63]] = [n, n - 5, n]
    a0 = gpu.from_numpy(few).cuda()
    a = a0.repeat(batch // 64 + 1, 1, 1)[:batch].contiguous()
    b0 = gpu.from_numpy(wl.rhs_rows(64, m, n, seed=6, ld=m)).cuda()
    b = b0.repeat(batch // 64 + 1, 1, 1)[:batch].contiguous()
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    kb.lib().kblas_posv_batch_strided_wsquery(handle.ptr, b"R", m, n, 1)
    assert handle.allocate_workspace() == 1
    if form == "strided":
        st = handle.call("kblasDposv_batch_strided", "R", "L", m, n, a.data_ptr(), n, n * n, b.data_ptr(),
                         m, n * m, batch, info.data_ptr())
    else:
        pa, pb = ptr_array(gpu, a), ptr_array(gpu, b)
        st = handle.call("kblasDposv_batch", "R", "L", m, n, pa.data_ptr(), n, pb.data_ptr(), m, batch,
                         info.data_ptr())
    assert st == 1
    gpu.cuda.synchronize()
    w = gpu.from_numpy(want).cuda().repeat(batch // 64 + 1)[:batch]
    assert bool((info == w).all())
    ok = w == 0
    # copies agree, in either slice; failed systems keep their right-hand sides
    same = lambda x: bool((x == x[:64].repeat(batch // 64 + 1, 1, 1)[:batch])[ok].all())
    assert same(a) and same(b)
    assert bool((b[~ok] == b0.repeat(batch // 64 + 1, 1, 1)[:batch][~ok]).all())
