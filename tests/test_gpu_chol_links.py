"""Double-precision POSV of strongly coupled groups of unknowns that single weak
couplings join: a component of a solution in one group for a right-hand side in another
hangs on the entry between them alone. Systems, references and bars (those of an FP64
Cholesky factorization, entry by entry and component by component) as in
test_gpu_chol_weak.py."""
import numpy as np
import pytest

from test_gpu_chol_weak import LD, U, chol_ld, cm, mul_ld, posv, solve_ld

pytestmark = pytest.mark.gpu


def groups(kind, n, v, rng):
    """Dense shifted blocks, neighbouring ones joined by one entry, v of its scale; in the
    last column of its block, so that L has no further entry between the two."""
    cut = {"halves": [n // 2], "quarter": [n // 4], "last": [n - 6], "three": [n // 3, 2 * n // 3]}[kind]
    a = np.zeros((n, n))
    ends = [0] + cut + [n]
    for lo, hi in zip(ends[:-1], ends[1:]):
        g = rng.standard_normal((hi - lo, hi - lo))
        a[lo:hi, lo:hi] = g @ g.T + (hi - lo) * np.eye(hi - lo)
    for c, hi in zip(cut, ends[2:]):
        i, j = rng.integers(c, hi), c - 1
        a[i, j] = a[j, i] = v * np.sqrt(a[i, i] * a[j, j])
    return a


@pytest.mark.parametrize("kind,v", [("halves", 1e-12), ("halves", 1e-5), ("quarter", 1e-9),
                                    ("last", 1e-12), ("three", 1e-7)])
@pytest.mark.parametrize("n,form,batch", [(32, "strided", 2), (64, "strided", 2), (100, "strided", 2),
                                          (110, "vbatch", 2), (120, "strided", 320),
                                          (160, "strided", 2)])
def test_joined_groups(gpu, handle, kb, kind, v, n, form, batch):
    mats = [groups(kind, n, v, np.random.default_rng(11 * n + s)) for s in range(2)]
    b = np.zeros((2, n, 2))
    b[:, 0, 0] = b[:, n - 1, 1] = 1.0
    k = batch // 2
    out, X = posv(gpu, handle, kb, np.tile(cm(mats), (k, 1, 1)), np.tile(b, (k, 1, 1)), form)
    for s, A in enumerate(mats):
        assert np.array_equal(out[s::2], np.tile(out[s], (k, 1, 1)))
        assert np.array_equal(X[s::2], np.tile(X[s], (k, 1, 1)))
        L = np.tril(out[s].T).astype(LD)
        scale = mul_ld(np.abs(L), np.abs(L).T)
        assert (np.abs(A - mul_ld(L, L.T)) <= (n + 8) * U * scale).all()
        R = chol_ld(A)
        inv = np.abs(solve_ld(R, np.eye(n)))
        for r in range(2):
            x = solve_ld(R, b[s, :, r])
            got = X[s, :, r].astype(LD)
            bar = (3 * n + 16) * U * 1.125 * mul_ld(inv, mul_ld(scale, np.abs(got)[:, None]))[:, 0]
            assert (np.abs(x - got) <= bar + LD(2.0 ** -1022)).all(), (s, r)
