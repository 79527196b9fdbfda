"""Double-precision products with short sums in the kernel that cuts its operands: matrices
of a variable-size batch with k below 16 next to larger ones, and uniform k with a
remainder of 1..15 beyond chunks of 64.

Bar for alpha = 1, beta = 0, that of a chain of FP64 FMAs: entry by entry
|C - op(A) op(B)| <= k u |op(A)| |op(B)| (u = 2^-53; the first of the k operations rounds a
product, the others a product and sum), with one more rounding per further chunk of the
sum. Reference in long double (IEEE quad on the GPU machine's Arm host, 64 bits of
mantissa elsewhere: 2^-11 of the bar)."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.longdouble


def product(a, b):
    out = np.zeros((a.shape[0], b.shape[1]), LD)
    for k in range(a.shape[1]):
        out += np.outer(a[:, k].astype(LD), b[k].astype(LD))
    return out


def check(got, a, b):
    k = a.shape[1]
    bar = (k + (k - 1) // 48) * U * 1.001 * product(np.abs(a), np.abs(b))
    assert (np.abs(got - product(a, b)) <= bar).all(), (a.shape, b.shape)


@pytest.mark.parametrize("tt", ["NN", "TT"])
def test_vbatch_short_k(gpu, handle, tt):
    ta, tb = tt
    rng = np.random.default_rng(3)
    ks = [1, 2, 3, 5, 7, 8, 9, 12, 15, 16, 17, 64, 65, 79, 100]
    ms = [1, 70, 64, 33, 65, 5, 40, 64, 31, 20, 64, 33, 66, 40, 100]
    ns = [1, 50, 32, 33, 31, 70, 40, 64, 9, 20, 32, 40, 33, 64, 100]
    A = [rng.standard_normal((k, m) if ta == "N" else (m, k)) for m, k in zip(ms, ks)]
    B = [rng.standard_normal((n, k) if tb == "N" else (k, n)) for n, k in zip(ns, ks)]
    dA, dB = [to_dev(gpu, x) for x in A], [to_dev(gpu, x) for x in B]
    dC = [gpu.full((n, m), float("nan"), dtype=gpu.float64, device="cuda") for m, n in zip(ms, ns)]
    ptrs = lambda ts: gpu.tensor([t.data_ptr() for t in ts], dtype=gpu.int64, device="cuda")
    ints = lambda v: gpu.tensor(v, dtype=gpu.int32, device="cuda")
    dm, dn, dk = ints(ms), ints(ns), ints(ks)
    pa, pb, pc = ptrs(dA), ptrs(dB), ptrs(dC)
    lda, ldb = (dm if ta == "N" else dk), (dk if tb == "N" else dn)
    assert handle.call("kblasDgemm_vbatch", ta, tb, dm.data_ptr(), dn.data_ptr(), dk.data_ptr(), 100, 100,
                       100, 1.0, pa.data_ptr(), lda.data_ptr(), pb.data_ptr(), ldb.data_ptr(), 0.0,
                       pc.data_ptr(), dm.data_ptr(), len(ks)) == 1
    gpu.cuda.synchronize()
    assert handle.device_status() == 1
    for i in range(len(ks)):
        a = A[i].T if ta == "N" else A[i]
        b = B[i].T if tb == "N" else B[i]
        check(dC[i].cpu().numpy().T, a, b)


@pytest.mark.parametrize("k", [16, 63, 65, 72, 79, 80, 129, 143, 193])
def test_remainders(gpu, handle, k):
    m, n = 70, 33
    rng = np.random.default_rng(k)
    A, B = rng.standard_normal((2, k, m)), rng.standard_normal((2, n, k))
    dA, dB = to_dev(gpu, A), to_dev(gpu, B)
    C = gpu.full((2, n, m), float("nan"), dtype=gpu.float64, device="cuda")
    assert handle.call("kblasDgemm_batch_strided", "N", "N", m, n, k, 1.0, dA.data_ptr(), m, m * k,
                       dB.data_ptr(), k, n * k, 0.0, C.data_ptr(), m, m * n, 2) == 1
    gpu.cuda.synchronize()
    for s in range(2):
        check(C[s].cpu().numpy().T, A[s].T, B[s].T)
