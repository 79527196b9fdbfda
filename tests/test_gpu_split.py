"""GPU parity of the double-precision products that run on the tensor cores by
exact slicing (GEMM and SYRK at the edges of their 64 x 32 tiles and 64-deep k
chunks), and of the data that the slicing hands back to FP64 FMAs: rows graded
over k, sparse operands, infinities and NaNs.

Bar: elementwise 10 k eps (|alpha| |op(A)| |op(B)| + |beta| |C|), the bound of
the FP64 kernels: the slicing drops at most (6 + 2) 2^-56 2^(Ei + Ej) per k and
every entry whose |op(A)| |op(B)| is below 2^-2 2^(Ei + Ej) (as estimated within
a factor of 2) is computed again, so an entry is off by at most about
8 k eps of it; a k chunk adds one rounding of C."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def run_gemm(gpu, handle, ta, tb, A, B, C, m, n, k, alpha, beta, form):
    lda, ldb, ldc = A.shape[2], B.shape[2], C.shape[2]
    batch = A.shape[0]
    dA, dB, dC = to_dev(gpu, A), to_dev(gpu, B), to_dev(gpu, C)
    if form == "strided":
        st = handle.call("kblasDgemm_batch_strided", ta, tb, m, n, k, alpha, dA.data_ptr(), lda,
                         A.shape[1] * lda, dB.data_ptr(), ldb, B.shape[1] * ldb, beta,
                         dC.data_ptr(), ldc, C.shape[1] * ldc, batch)
    else:
        pa, pb, pc = ptr_array(gpu, dA), ptr_array(gpu, dB), ptr_array(gpu, dC)
        st = handle.call("kblasDgemm_batch", ta, tb, m, n, k, alpha, pa.data_ptr(), lda,
                         pb.data_ptr(), ldb, beta, pc.data_ptr(), ldc, batch)
    assert st == 1
    gpu.cuda.synchronize()
    assert handle.device_status() == 1
    return dC.cpu().numpy()


def operands(rng, batch, ta, tb, m, n, k, pad):
    A = rng.standard_normal((batch, k if ta == "N" else m, (m if ta == "N" else k) + pad))
    B = rng.standard_normal((batch, n if tb == "N" else k, (k if tb == "N" else n) + pad))
    return A, B


def dense_ops(A, B, ta, tb, m, n, k):
    a = A[:, :, :m].transpose(0, 2, 1) if ta == "N" else A[:, :, :k]
    b = B[:, :, :k].transpose(0, 2, 1) if tb == "N" else B[:, :, :n]
    return a, b


@pytest.mark.parametrize("mnk", [(24, 24, 16), (63, 31, 63), (64, 32, 64), (65, 33, 65),
                                 (16, 129, 31), (129, 20, 128), (200, 70, 193)])
@pytest.mark.parametrize("tt", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("pad,form", [(0, "strided"), (1, "array")])
def test_gemm_tile_edges(gpu, handle, mnk, tt, pad, form):
    m, n, k = mnk
    ta, tb = tt
    rng = np.random.default_rng(m + 7 * n + 11 * k + pad)
    A, B = operands(rng, 3, ta, tb, m, n, k, pad)
    C = rng.standard_normal((3, n, m + pad))
    out = run_gemm(gpu, handle, ta, tb, A, B, C, m, n, k, 1.25, -0.5, form)
    assert np.array_equal(out[:, :, m:], C[:, :, m:])
    a, b = dense_ops(A, B, ta, tb, m, n, k)
    want = 1.25 * (a @ b) - 0.5 * C[:, :, :m].transpose(0, 2, 1)
    scale = 1.25 * (np.abs(a) @ np.abs(b)) + 0.5 * np.abs(C[:, :, :m].transpose(0, 2, 1))
    got = out[:, :, :m].transpose(0, 2, 1)
    assert (np.abs(got - want) <= 10 * k * U * scale).all()


@pytest.mark.parametrize("data", ["graded_k", "graded_rows", "sparse", "near_power_of_two", "tiny",
                                  "zero_rows"])
def test_gemm_hard_data(gpu, handle, data):
    m, n, k = 70, 40, 100
    rng = np.random.default_rng(len(data))
    A, B = operands(rng, 4, "N", "N", m, n, k, 0)  # A[b, l, i], B[b, j, l]
    if data == "graded_k":
        d = 10.0 ** np.linspace(0, 16, k)
        A *= d[None, :, None]
        B /= d[None, None, :]
    elif data == "graded_rows":
        A *= (10.0 ** np.linspace(-60, 60, m))[None, None, :]
        B *= (10.0 ** np.linspace(40, -40, n))[None, :, None]
    elif data == "sparse":
        A[rng.random(A.shape) < 0.9] = 0.0
        B[rng.random(B.shape) < 0.9] = 0.0
    elif data == "near_power_of_two":  # first digits at the end of their range
        A = np.sign(A) * (2.0 - 2.0 ** -rng.integers(3, 50, A.shape))
        B = np.sign(B) * (2.0 - 2.0 ** -rng.integers(3, 50, B.shape))
    elif data == "tiny":
        A *= 1e-155
        B *= 1e-150
    else:
        A[:, :, ::3] = 0.0
        B[:, ::2, :] = 0.0
    C = np.full((4, n, m), np.nan)  # beta = 0: not read
    out = run_gemm(gpu, handle, "N", "N", A, B, C, m, n, k, 1.0, 0.0, "strided")
    a, b = dense_ops(A, B, "N", "N", m, n, k)
    want, scale = a @ b, np.abs(a) @ np.abs(b)
    assert (np.abs(out.transpose(0, 2, 1) - want) <= 10 * k * U * scale).all()


def test_gemm_infinities_and_nans(gpu, handle):
    m, n, k = 66, 50, 70
    rng = np.random.default_rng(3)
    A, B = operands(rng, 3, "N", "N", m, n, k, 0)
    A[0, 5, 3], A[1, 69, 65], B[2, 7, 66] = np.nan, np.inf, -np.inf
    C = rng.standard_normal((3, n, m))
    out = run_gemm(gpu, handle, "N", "N", A, B, C, m, n, k, 1.0, 1.0, "strided")
    a, b = dense_ops(A, B, "N", "N", m, n, k)
    with np.errstate(invalid="ignore"):
        want = C.transpose(0, 2, 1) + a @ b
    got = out.transpose(0, 2, 1)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf])
    fin = np.isfinite(want)
    assert np.abs(got[fin] - want[fin]).max() <= 10 * k * U * 1e3


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("mk", [(24, 16), (64, 64), (65, 63), (97, 65), (160, 130)])
def test_syrk_tile_edges(gpu, handle, uplo, trans, mk):
    m, k = mk
    batch = 5
    rng = np.random.default_rng(m + k)
    A = rng.standard_normal((batch, k, m) if trans == "N" else (batch, m, k))
    C = rng.standard_normal((batch, m, m))
    dA, dC = to_dev(gpu, A), to_dev(gpu, C)
    assert handle.call("kblasDsyrk_batch_strided", uplo, trans, m, k, -1.0, dA.data_ptr(),
                       A.shape[2], m * k, 1.0, dC.data_ptr(), m, m * m, batch) == 1
    gpu.cuda.synchronize()
    a = A.transpose(0, 2, 1) if trans == "N" else A
    want = C.transpose(0, 2, 1) - a @ a.transpose(0, 2, 1)
    scale = np.abs(C.transpose(0, 2, 1)) + np.abs(a) @ np.abs(a).transpose(0, 2, 1)
    got = dC.cpu().numpy().transpose(0, 2, 1)
    keep = np.tril(np.ones((m, m), bool)) if uplo == "L" else np.triu(np.ones((m, m), bool))
    assert (np.abs(got - want) <= 10 * k * U * scale)[:, keep].all()
    assert np.array_equal(got[:, ~keep], C.transpose(0, 2, 1)[:, ~keep])
