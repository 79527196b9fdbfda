"""Double-precision POTRF / POSV entry by entry: matrices whose couplings lie far below
their diagonals, and the accuracy of the ones that stay in fixed point.

References in long double (IEEE quad on the GPU machine's Arm host, 64 bits of mantissa
elsewhere). Bars for the factor and the solutions of weakly coupled unknowns, those of
an FP64 Cholesky factorization (u = 2^-53; the reciprocal pivots' roundings are in the
added constant):
  |A - L L^T| <= (n + 8) u |L| |L^T|                       entry by entry,
  |x - X|     <= (3 n + 16) u |A^-1| |L| |L^T| |X| (1 + 1/8) component by component,
and the smallest normal number, 2^-1022: components below it have no FP64 value.
A matrix that stays in fixed point has in addition, from entries rounded to 2^-60 of
their rows' scales 2^E <= 2.01 sqrt(a_ii) and a product of low limbs (2^-60) dropped
per column, (n + 4 sqrt(n) + 8) 2^-60 2^(E_i + E_j), and its root mean square error
relative to |L| |L^T| is at most twice that of the oracle's FP64 factor."""
import numpy as np
import pytest

from gpu_util import ptr_array, to_dev

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.longdouble


def chol_ld(A):
    n = A.shape[0]
    S, L = A.astype(LD), np.zeros((n, n), LD)
    for k in range(n):
        L[k:, k] = S[k:, k] / np.sqrt(S[k, k])
        S[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], L[k + 1:, k])
    return L


def solve_ld(L, b):
    n = L.shape[0]
    x = b.astype(LD)
    for k in range(n):
        x[k] = x[k] / L[k, k]
        x[k + 1:] -= (L[k + 1:, k] if x.ndim == 1 else L[k + 1:, k:k + 1]) * x[k]
    for k in range(n - 1, -1, -1):
        x[k] = x[k] / L[k, k]
        x[:k] -= (L[k, :k] if x.ndim == 1 else L[k, :k, None]) * x[k]
    return x


def mul_ld(X, Y):
    out = np.zeros((X.shape[0], Y.shape[1]), LD)
    for k in range(X.shape[1]):
        out += np.outer(X[:, k], Y[k])
    return out


def sym(n, rng, e):
    a = np.tril(rng.standard_normal((n, n)) * e, -1)
    return a + a.T + np.eye(n)


def cov(n, rng, ell):
    p = rng.uniform(0, 1, (n, 2))
    d2 = ((p[:, None] - p[None]) ** 2).sum(-1)
    return np.exp(-d2 / (2 * ell * ell)) + 1e-4 * np.eye(n)


def weak(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind.startswith("tri"):
        return np.eye(n) + float(kind[3:]) * (np.eye(n, k=1) + np.eye(n, k=-1))
    if kind.startswith("dense"):
        return sym(n, rng, float(kind[5:]))
    if kind.startswith("cov"):
        return cov(n, rng, float(kind[3:]))
    g = rng.standard_normal((n, n))
    a = g @ g.T + n * np.eye(n)
    if kind == "one":  # one unknown coupled by 1e-10, neither first nor last
        k = n // 3
        a[k, :k] *= 1e-10
        a[k, k + 1:] *= 1e-10
        a[:, k] = a[k]
    elif kind == "blocks":  # two halves coupled by 1e-12
        h = n // 2
        a[h:, :h] *= 1e-12
        a[:h, h:] = a[h:, :h].T
    elif kind == "grid":  # five-point stencil with a strong diagonal: the fill decays
        w = max(3, int(np.sqrt(n)))
        a = 100.0 * np.eye(n)
        i = np.arange(n)
        r = i[(i + 1 < n) & ((i + 1) % w != 0)]
        a[r, r + 1] = a[r + 1, r] = -1.0
        r = i[i + w < n]
        a[r, r + w] = a[r + w, r] = -1.0
    return a


def cm(mats):
    """(batch, n, n) column-major batch of symmetric matrices."""
    return np.ascontiguousarray(np.stack(mats).transpose(0, 2, 1))


def posv(gpu, handle, kb, a, b, form="strided"):
    batch, n, m = b.shape
    da, db = to_dev(gpu, a), to_dev(gpu, b)
    info = gpu.full((batch,), -99, dtype=gpu.int32, device="cuda")
    if form == "strided":
        kb.lib().kblas_posv_batch_strided_wsquery(handle.ptr, b"R", m, n, batch)
        assert handle.allocate_workspace() == 1
        st = handle.call("kblasDposv_batch_strided", "R", "L", m, n, da.data_ptr(), n, n * n,
                         db.data_ptr(), m, n * m, batch, info.data_ptr())
    else:
        kb.lib().kblas_posv_vbatch_wsquery(handle.ptr, n, batch)
        assert handle.allocate_workspace() == 1
        pa, pb = ptr_array(gpu, da), ptr_array(gpu, db)
        full = lambda v: gpu.full((batch,), v, dtype=gpu.int32, device="cuda")
        dm, dn = full(m), full(n)
        st = handle.call("kblasDposv_vbatch", "R", "L", dm.data_ptr(), dn.data_ptr(), m, n,
                         pa.data_ptr(), dn.data_ptr(), pb.data_ptr(), dm.data_ptr(), batch,
                         info.data_ptr())
    assert st == 1
    gpu.cuda.synchronize()
    assert handle.device_status() == 1
    assert (info.cpu().numpy() == 0).all()
    return da.cpu().numpy(), db.cpu().numpy()


KINDS = ["tri1e-14", "tri1e-5", "dense1e-8", "dense1e-10", "dense1e-18", "cov0.05", "cov0.1",
         "one", "blocks", "grid"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,form", [(20, "strided"), (32, "strided"), (48, "strided"),
                                    (48, "vbatch"), (110, "strided")])
def test_weak_couplings(gpu, handle, kb, kind, n, form):
    mats = [weak(kind, n, 7 * n + s) for s in range(2)]
    # unit right-hand sides at both ends and a general one
    b = np.zeros((2, n, 3))
    b[:, 0, 0] = b[:, n - 1, 1] = 1.0
    b[:, :, 2] = np.random.default_rng(n).standard_normal((2, n))
    out, X = posv(gpu, handle, kb, cm(mats), b, form)
    for s, A in enumerate(mats):
        L = np.tril(out[s].T).astype(LD)
        scale = mul_ld(np.abs(L), np.abs(L).T)
        assert (np.abs(A - mul_ld(L, L.T)) <= (n + 8) * U * scale).all()
        R = chol_ld(A)
        inv = np.abs(solve_ld(R, np.eye(n)))
        for r in range(3):
            x = solve_ld(R, b[s, :, r])
            got = X[s, :, r].astype(LD)
            bar = (3 * n + 16) * U * 1.125 * mul_ld(inv, mul_ld(scale, np.abs(got)[:, None]))[:, 0]
            bar = bar + LD(2.0 ** -1022)
            assert (np.abs(x - got) <= bar).all(), (s, r)


@pytest.mark.parametrize("kind", ["shifted", "cov0.3"])
@pytest.mark.parametrize("n", [20, 64, 128, 150])
def test_fixed_point_entries(gpu, handle, kb, orc, kind, n):
    mats = [weak(kind, n, 5 * n + s) for s in range(2)]
    b = np.zeros((2, n, 1))
    out, _ = posv(gpu, handle, kb, cm(mats), b)
    ref = cm(mats)
    assert (orc.potrf_batch(ref, n) == 0).all()
    for s, A in enumerate(mats):
        R = np.abs(chol_ld(A))
        scale = mul_ld(R, R.T)
        low = np.tril_indices(n)
        rms = []
        for F in (out[s], ref[s]):
            L = np.tril(F.T).astype(LD)
            e = np.abs(A - mul_ld(L, L.T))
            rms.append(np.sqrt(np.mean((e / scale)[low].astype(float) ** 2)))
            if F is out[s]:
                d = 2.01 * np.sqrt(np.diag(A))
                bar = (n + 8) * U * scale + (n + 4 * np.sqrt(n) + 8) * 2.0 ** -60 * np.outer(d, d)
                assert (e <= bar).all()
        assert rms[0] <= 2 * rms[1], rms
