"""TRSM / TRMM at the edges of the staged triangle's groups of four rows (remainders of
0..3 rows, one group and none) and at the orders where the staged form is largest, double
and complex double, against the oracle's or a dense product; bar of test_gpu_tri.py's kind:
componentwise backward error, |op(A) X - B| <= 2 (K + 4) u' |op(A)| |X| for TRSM and
|X - op(A) B| <= 2 (K + 4) u' |op(A)| |B| for TRMM, half of it the check's own rounding (u' = 2^-53, four times that for complex
products), K the triangle's order."""
import numpy as np
import pytest

from gpu_util import to_dev

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def triangle(rng, k, lower, cplx):
    a = rng.standard_normal((k, k)) / np.sqrt(k)
    if cplx:
        a = a + 1j * rng.standard_normal((k, k)) / np.sqrt(k)
    a = np.tril(a, -1) + np.diag(rng.uniform(1, 2, k))
    return a if lower else a.T.copy()


@pytest.mark.parametrize("op", ["trsm", "trmm"])
@pytest.mark.parametrize("prec,k", [("D", k) for k in (1, 2, 3, 4, 5, 6, 7, 8, 9, 115, 116, 117, 118, 127)]
                         + [("Z", k) for k in (1, 3, 4, 5, 70, 71, 89, 90)])
@pytest.mark.parametrize("side,uplo,trans", [("L", "L", "N"), ("L", "U", "N"), ("R", "L", "N"), ("R", "U", "T")])
def test_groups(gpu, handle, op, prec, k, side, uplo, trans):
    cplx = prec == "Z"
    rng = np.random.default_rng(k)
    vecs, batch, alpha = 67, 3, 1.0
    A = np.stack([triangle(rng, k, uplo == "L", cplx) for _ in range(batch)])
    m, n = (k, vecs) if side == "L" else (vecs, k)
    B = rng.standard_normal((batch, m, n))
    if cplx:
        B = B + 1j * rng.standard_normal((batch, m, n))
    other = np.triu(np.ones((k, k), bool), 1) if uplo == "L" else np.tril(np.ones((k, k), bool), -1)
    stored = np.where(other, np.nan, A)           # the other triangle is not read
    dA = to_dev(gpu, stored.transpose(0, 2, 1))
    dB = to_dev(gpu, B.transpose(0, 2, 1))
    assert handle.call(f"kblas{prec}{op}_batch_strided", side, uplo, trans, "N", m, n, alpha, dA.data_ptr(),
                       k, k * k, dB.data_ptr(), m, m * n, batch) == 1
    gpu.cuda.synchronize()
    X = dB.cpu().numpy().transpose(0, 2, 1)
    u = 4 * U if cplx else U
    for s in range(batch):
        M = A[s].T if trans == "T" else A[s]
        mul = (lambda p, q: p @ q) if side == "L" else (lambda p, q: q @ p)
        if op == "trsm":
            err, scale = np.abs(mul(M, X[s]) - B[s]), mul(np.abs(M), np.abs(X[s]))
        else:
            err, scale = np.abs(X[s] - mul(M, B[s])), mul(np.abs(M), np.abs(B[s]))
        # the check's own product rounds as often
        assert (err <= 2 * (k + 4) * u * scale).all()
