"""Performance cases: the batched Cholesky / triangular work a user of the library runs.

Every case is a dict of plain values with a ``kind``:

  posv          DPOSV / SPOSV, uniform order (factor + solve, info)
  potrf_potrs   DPOTRF then DPOTRS (a factor that is kept and solved with)
  trsm, trmm    triangular solve / product, every side, uplo and trans
  syrk          symmetric rank-k update, lower or upper, N or T
  gemm_vbatch   variable-size GEMM (pointer arrays, per-matrix m, n, k)
  mixed         mixed-precision DPOSV, uniform order
  vbatch        variable-size DPOSV (pointer arrays), plain FP64 or mixed precision

The routines work in place. As in a program that refills its buffers between
calls, one pass first copies the operands it overwrites from the state's own
copy and then makes the call. Matrices are column-major: a tensor of shape
(batch, columns, ld) holds element (i, j) of matrix b at [b, j, i].
"""
import importlib
import math

import numpy as np
import torch

DT = {"d": torch.float64, "s": torch.float32}


def _lib():
    return importlib.import_module("kblas-gpu_gb300")


def listed():
    return [
        # a small call inside a host loop (a filter's 200 covariance updates): latency
        {"name": "posv_small", "kind": "posv", "prec": "d", "n": 24, "m": 1, "batch": 200,
         "form": "strided", "recipe": "shifted"},
        # many small systems, the factor kept: the uniform benchmark configuration
        {"name": "potrf_potrs_n32", "kind": "potrf_potrs", "prec": "d", "n": 32, "m": 1,
         "batch": 10000, "form": "strided", "recipe": "shifted"},
        # single precision, an order that is no multiple of the block, pointer arrays
        {"name": "posv_s_n100", "kind": "posv", "prec": "s", "n": 100, "m": 3, "batch": 4000,
         "form": "array", "recipe": "shifted"},
        # one block order of conditioned systems with a few right-hand sides
        {"name": "posv_d_n64", "kind": "posv", "prec": "d", "n": 64, "m": 4, "batch": 20000,
         "form": "strided", "recipe": "cond"},
        # the building blocks of tile algorithms: 64 x 64 tiles
        {"name": "trsm_n64", "kind": "trsm", "prec": "d", "side": "L", "uplo": "L", "trans": "N",
         "m": 64, "n": 64, "batch": 20000, "form": "strided"},
        {"name": "trmm_n64", "kind": "trmm", "prec": "d", "side": "L", "uplo": "L", "trans": "N",
         "m": 64, "n": 64, "batch": 20000, "form": "array"},
        {"name": "syrk_n64", "kind": "syrk", "prec": "d", "uplo": "L", "trans": "N", "m": 64,
         "k": 64, "batch": 20000, "form": "strided"},
        # updates between blocks of uneven size (a multifrontal or low-rank tile code)
        {"name": "gemm_vbatch", "kind": "gemm_vbatch", "prec": "d", "lo": 16, "hi": 128,
         "transa": "N", "transb": "T", "batch": 8000},
        # mixed precision on large uniform systems (well conditioned: what it is meant for)
        {"name": "mixed_n400", "kind": "mixed", "n": 400, "m": 4, "batch": 300},
        # the variable-size batch of the headline, both precisions, 1% indefinite
        {"name": "vbatch_mixed", "kind": "vbatch", "mixed": True, "nmin": 8, "nmax": 256,
         "batch": 30000},
        {"name": "vbatch_fp64", "kind": "vbatch", "mixed": False, "nmin": 8, "nmax": 256,
         "batch": 20000},
        # covariance matrices of spatial statistics, ill conditioned, 8 right-hand sides
        {"name": "posv_cov_n512", "kind": "posv", "prec": "d", "n": 512, "m": 8, "batch": 500,
         "form": "strided", "recipe": "cov"},
    ]


def _logint(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["posv", "posv", "potrf_potrs", "trsm", "trmm", "syrk", "gemm_vbatch",
                       "mixed", "vbatch", "vbatch"])
    form = rng.choice(["strided", "array"])
    prec = rng.choice(["d", "d", "s"])

    def batch_for(flops, bytes_, most=20000):
        top = max(50, int(min(most, 1.0e10 / flops, 1.0e9 / bytes_)))
        return _logint(rng, 50, top)

    if kind in ("posv", "potrf_potrs"):
        n, m = _logint(rng, 4, 400), _logint(rng, 1, 8)
        return {"kind": kind, "prec": prec, "n": n, "m": m,
                "batch": batch_for(n ** 3 / 3 + 4 * n * n * m, 16 * n * n), "form": form,
                "recipe": rng.choice(["shifted", "cov"]) if prec == "d" and n >= 32 else "shifted"}
    if kind in ("trsm", "trmm"):
        m, n = _logint(rng, 8, 200), _logint(rng, 8, 200)
        side = rng.choice(["L", "R"])
        k = m if side == "L" else n
        return {"kind": kind, "prec": prec, "side": side, "uplo": rng.choice(["L", "L", "U"]),
                "trans": rng.choice(["N", "T"]), "m": m, "n": n,
                "batch": batch_for(4 * m * n * k, 8 * (k * k + 2 * m * n)), "form": form}
    if kind == "syrk":
        m, k = _logint(rng, 8, 200), _logint(rng, 8, 200)
        return {"kind": kind, "prec": prec, "uplo": rng.choice(["L", "L", "U"]),
                "trans": rng.choice(["N", "T"]), "m": m, "k": k,
                "batch": batch_for(2 * m * m * k, 8 * (k * m + 2 * m * m)), "form": form}
    if kind == "gemm_vbatch":
        lo = _logint(rng, 8, 32)
        hi = _logint(rng, 2 * lo, 160)
        return {"kind": kind, "prec": prec, "lo": lo, "hi": hi, "transa": rng.choice(["N", "T"]),
                "transb": rng.choice(["N", "T"]), "batch": batch_for(2 * hi ** 3, 24 * hi * hi, 10000)}
    if kind == "mixed":
        n, m = _logint(rng, 16, 400), _logint(rng, 1, 6)
        return {"kind": kind, "n": n, "m": m,
                "batch": batch_for(n ** 3 / 3 + 8 * n * n * m, 8 * n * n)}
    nmax = _logint(rng, 32, 256)
    return {"kind": "vbatch", "mixed": rng.random() < 0.5, "nmin": _logint(rng, 4, 16),
            "nmax": nmax, "batch": batch_for(nmax ** 3 / 9, 4 * nmax * nmax)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 + seed)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _spd(g, recipe, batch, n):
    """(batch, n, n) symmetric positive definite, FP64."""
    out = torch.empty(batch, n, n, dtype=torch.float64, device="cuda")
    step = max(1, int(4.0e7 // (n * n)))
    for c in range(0, batch, step):
        k = min(step, batch - c)
        if recipe == "shifted":
            # G G^T + n I
            x = _randn(g, k, n, n)
            a = x @ x.transpose(1, 2)
            a.diagonal(dim1=1, dim2=2).add_(float(n))
        elif recipe == "cond":
            # Q diag(lambda) Q^T, condition numbers log-uniform in [1e2, 1e6]
            p = torch.rand(k, 1, generator=g, dtype=torch.float64, device="cuda") * 4 + 2
            t = torch.linspace(0, 1, n, dtype=torch.float64, device="cuda")
            a = torch.diag_embed(10.0 ** (-p * t))
            for _ in range(3):
                v = _randn(g, k, n, 1)
                v = v / v.norm(dim=1, keepdim=True)
                a = a - 2 * v @ (v.transpose(1, 2) @ a)
                a = a - 2 * (a @ v) @ v.transpose(1, 2)
            a = 0.5 * (a + a.transpose(1, 2))
        else:
            # squared-exponential covariance of n points in the unit square
            xy = torch.rand(k, 2, n, generator=g, dtype=torch.float64, device="cuda")
            ell = torch.rand(k, 1, 1, generator=g, dtype=torch.float64, device="cuda") * 0.25 + 0.05
            d2 = (xy[:, 0, :, None] - xy[:, 0, None, :]) ** 2
            d2 += (xy[:, 1, :, None] - xy[:, 1, None, :]) ** 2
            a = torch.exp(-d2 / (2 * ell * ell))
            a.diagonal(dim1=1, dim2=2).add_(1e-4)
        out[c:c + k] = a
    return out


def _tri(g, batch, k, uplo, prec):
    """Triangular factors, column-major; the other triangle is zero."""
    a = _randn(g, batch, k, k) / math.sqrt(k)
    a = torch.tril(a, -1)
    a.diagonal(dim1=1, dim2=2).copy_(
        torch.rand(batch, k, generator=g, dtype=torch.float64, device="cuda") + 1.0)
    # a[b] row-major lower; a column-major lower matrix is stored transposed
    return (a.transpose(1, 2) if uplo == "L" else a).contiguous().to(DT[prec])


def _vsizes(batch, lo, hi):
    # the orders belong to the case (a user's mesh or tree), the values to the seed
    u = np.random.default_rng(77).uniform(math.log(lo), math.log(hi + 1), batch)
    return np.clip(np.floor(np.exp(u)).astype(np.int32), lo, hi)


def _vpool(case, seed):
    """Sizes, pool of SPD matrices grouped by order (the indefinite 1% last) and offsets."""
    g = _gen(seed)
    batch = case["batch"]
    ns = _vsizes(batch, case["nmin"], case["nmax"])
    bad = np.zeros(batch, bool)
    bad[::100] = True
    order = np.lexsort((ns, bad))
    sz = ns.astype(np.int64) ** 2
    offs = np.zeros(batch, np.int64)
    offs[order] = np.concatenate([[0], np.cumsum(sz[order])[:-1]])
    pool = torch.empty(int(sz.sum()), dtype=torch.float64, device="cuda")
    k = 0
    while k < batch:
        n, isbad = int(ns[order[k]]), bool(bad[order[k]])
        e = k
        while e < batch and ns[order[e]] == n and bad[order[e]] == isbad:
            e += 1
        a = _spd(g, "shifted", e - k, n)
        if isbad:
            # one negative direction: v^T A v changes its sign
            v = _randn(g, e - k, n, 1)
            v = v / v.norm(dim=1, keepdim=True)
            a = a - 2 * (v.transpose(1, 2) @ a @ v) * (v @ v.transpose(1, 2))
            a = 0.5 * (a + a.transpose(1, 2))
        o = int(offs[order[k]])
        pool[o:o + (e - k) * n * n] = a.reshape(-1)
        k = e
    bad_lo = int(offs[bad].min()) if bad.any() else int(sz.sum())
    boffs = np.concatenate([[0], np.cumsum(ns.astype(np.int64))[:-1]])
    b = _randn(g, int(ns.sum()))
    return ns, order, bad, offs, boffs, pool, b, bad_lo


def _gemm_sizes(case):
    r = np.random.default_rng(99)
    return [r.integers(case["lo"], case["hi"] + 1, case["batch"]).astype(np.int32) for _ in range(3)]


def _offs(sizes):
    return np.concatenate([[0], np.cumsum(sizes.astype(np.int64))[:-1]])


def _ptrs(t, offs):
    return torch.from_numpy(t.data_ptr() + np.asarray(offs, np.int64) * t.element_size()).cuda()


def _uptrs(t):
    return _ptrs(t, np.arange(t.shape[0], dtype=np.int64) * t.stride(0))


class _State:
    pass


def prepare(case, seed):
    kb = _lib()
    s = _State()
    s.case = case
    kind = case["kind"]
    s.h = h = kb.Handle()
    g = _gen(seed)
    p = case.get("prec", "d")
    batch = case["batch"]
    if kind in ("posv", "potrf_potrs", "mixed"):
        n, m = case["n"], case["m"]
        s.A0 = _spd(g, case.get("recipe", "shifted"), batch, n).to(DT[p])
        s.B0 = _randn(g, batch, n, m).to(DT[p])
        s.A, s.B = s.A0.clone(), s.B0.clone()
        s.info = torch.zeros(batch, dtype=torch.int32, device="cuda")
        if kind == "mixed":
            s.iter = torch.zeros(batch, dtype=torch.int32, device="cuda")
            kb.lib().kblas_posv_batch_mixed_wsquery(h.ptr, b"R", m, n, batch)
        elif kind == "posv":
            kb.lib().kblas_posv_batch_strided_wsquery(h.ptr, b"R", m, n, batch)
        else:
            kb.lib().kblas_potrf_batch_strided_wsquery(h.ptr, n, batch)
            kb.lib().kblas_potrs_batch_strided_wsquery(h.ptr, m, n, batch)
        if case.get("form") == "array":
            s.pA, s.pB = _uptrs(s.A), _uptrs(s.B)
    elif kind in ("trsm", "trmm"):
        m, n = case["m"], case["n"]
        k = m if case["side"] == "L" else n
        s.A = _tri(g, batch, k, case["uplo"], p)
        s.B0 = _randn(g, batch, n, m).to(DT[p])
        s.B = s.B0.clone()
        if case["form"] == "array":
            s.pA, s.pB = _uptrs(s.A), _uptrs(s.B)
    elif kind == "syrk":
        m, k = case["m"], case["k"]
        s.A = (_randn(g, batch, k, m) if case["trans"] == "N" else _randn(g, batch, m, k)).to(DT[p])
        s.C0 = _spd(g, "shifted", batch, m).to(DT[p])
        s.C = s.C0.clone()
        if case["form"] == "array":
            s.pA, s.pC = _uptrs(s.A), _uptrs(s.C)
    elif kind == "gemm_vbatch":
        m, n, k = _gemm_sizes(case)
        sa, sb, sc = m * k, k * n, m * n
        s.A = _randn(g, int(sa.sum())).to(DT[p])
        s.B = _randn(g, int(sb.sum())).to(DT[p])
        s.C0 = _randn(g, int(sc.sum())).to(DT[p])
        s.C = s.C0.clone()
        s.pA, s.pB, s.pC = _ptrs(s.A, _offs(sa)), _ptrs(s.B, _offs(sb)), _ptrs(s.C, _offs(sc))
        s.m, s.n, s.k = (torch.from_numpy(v).cuda() for v in (m, n, k))
        s.lda = s.m if case["transa"] == "N" else s.k
        s.ldb = s.k if case["transb"] == "N" else s.n
    else:
        ns, _, _, offs, boffs, pool, b, s.bad_lo = _vpool(case, seed)
        s.A, s.B0 = pool, b
        s.A0 = pool[s.bad_lo:].clone() if case["mixed"] else pool.clone()
        s.B = b.clone()
        s.pA, s.pB = _ptrs(s.A, offs), _ptrs(s.B, boffs)
        s.ns = torch.from_numpy(ns).cuda()
        s.ms = torch.ones(batch, dtype=torch.int32, device="cuda")
        s.ldb = torch.ones(batch, dtype=torch.int32, device="cuda")
        s.max_n = int(ns.max())
        s.info = torch.zeros(batch, dtype=torch.int32, device="cuda")
        s.iter = torch.zeros(batch, dtype=torch.int32, device="cuda")
        kb.lib().kblas_posv_vbatch_wsquery(h.ptr, s.max_n, batch)
    kb.check(h.allocate_workspace(), "kblasAllocateWorkspace")
    s.check = kb.check
    return s


def run(s):
    c, h = s.case, s.h
    kind, batch = c["kind"], c["batch"]
    P = c.get("prec", "d").upper()
    arr = c.get("form") == "array"
    if kind in ("posv", "potrf_potrs", "mixed"):
        n, m = c["n"], c["m"]
        s.A.copy_(s.A0)
        s.B.copy_(s.B0)
        if kind == "mixed":
            st = h.call("kblasDposv_batch_mixed_strided", "R", "L", m, n, s.A.data_ptr(), n, n * n,
                        s.B.data_ptr(), m, m * n, batch, s.info.data_ptr(), s.iter.data_ptr())
            s.check(st, "mixed posv")
            # iter reports how each system was refined; the results are X and info
            return {"x": s.B, "info": s.info}
        if kind == "posv":
            if arr:
                st = h.call(f"kblas{P}posv_batch", "R", "L", m, n, s.pA.data_ptr(), n,
                            s.pB.data_ptr(), m, batch, s.info.data_ptr())
            else:
                st = h.call(f"kblas{P}posv_batch_strided", "R", "L", m, n, s.A.data_ptr(), n, n * n,
                            s.B.data_ptr(), m, m * n, batch, s.info.data_ptr())
            s.check(st, "posv")
        elif arr:
            s.check(h.call(f"kblas{P}potrf_batch", "L", n, s.pA.data_ptr(), n, batch,
                           s.info.data_ptr()), "potrf")
            s.check(h.call(f"kblas{P}potrs_batch", "R", "L", m, n, s.pA.data_ptr(), n,
                           s.pB.data_ptr(), m, batch), "potrs")
        else:
            s.check(h.call(f"kblas{P}potrf_batch_strided", "L", n, s.A.data_ptr(), n, n * n, batch,
                           s.info.data_ptr()), "potrf")
            s.check(h.call(f"kblas{P}potrs_batch_strided", "R", "L", m, n, s.A.data_ptr(), n, n * n,
                           s.B.data_ptr(), m, m * n, batch), "potrs")
        return {"l": s.A, "x": s.B, "info": s.info}
    if kind in ("trsm", "trmm"):
        m, n = c["m"], c["n"]
        k = m if c["side"] == "L" else n
        s.B.copy_(s.B0)
        f = (c["side"], c["uplo"], c["trans"], "N", m, n, 1.0)
        if arr:
            st = h.call(f"kblas{P}{kind}_batch", *f, s.pA.data_ptr(), k, s.pB.data_ptr(), m, batch)
        else:
            st = h.call(f"kblas{P}{kind}_batch_strided", *f, s.A.data_ptr(), k, k * k,
                        s.B.data_ptr(), m, m * n, batch)
        s.check(st, kind)
        return s.B
    if kind == "syrk":
        m, k = c["m"], c["k"]
        lda = m if c["trans"] == "N" else k
        s.C.copy_(s.C0)
        if arr:
            st = h.call(f"kblas{P}syrk_batch", c["uplo"], c["trans"], m, k, -1.0, s.pA.data_ptr(),
                        lda, 1.0, s.pC.data_ptr(), m, batch)
        else:
            st = h.call(f"kblas{P}syrk_batch_strided", c["uplo"], c["trans"], m, k, -1.0,
                        s.A.data_ptr(), lda, m * k, 1.0, s.C.data_ptr(), m, m * m, batch)
        s.check(st, kind)
        return s.C
    if kind == "gemm_vbatch":
        s.C.copy_(s.C0)
        hi = c["hi"]
        st = h.call(f"kblas{P}gemm_vbatch", c["transa"], c["transb"], s.m.data_ptr(),
                    s.n.data_ptr(), s.k.data_ptr(), hi, hi, hi, -1.0, s.pA.data_ptr(),
                    s.lda.data_ptr(), s.pB.data_ptr(), s.ldb.data_ptr(), 1.0, s.pC.data_ptr(),
                    s.m.data_ptr(), batch)
        s.check(st, kind)
        return s.C
    # variable-size POSV; the mixed form leaves A as it is but for the systems
    # it solves in FP64 (here the indefinite ones, kept at the pool's end)
    (s.A[s.bad_lo:] if c["mixed"] else s.A).copy_(s.A0)
    s.B.copy_(s.B0)
    args = ["R", "L", s.ms.data_ptr(), s.ns.data_ptr(), 1, s.max_n, s.pA.data_ptr(),
            s.ns.data_ptr(), s.pB.data_ptr(), s.ldb.data_ptr(), batch, s.info.data_ptr()]
    if c["mixed"]:
        s.check(h.call("kblasDposv_vbatch_mixed", *args, s.iter.data_ptr()), kind)
        return {"x": s.B, "info": s.info}
    s.check(h.call("kblasDposv_vbatch", *args), kind)
    return {"l": s.A, "x": s.B, "info": s.info}


# ---------------------------------------------------------------- bounds, exact results
def work(case):
    kind, batch = case["kind"], case["batch"]
    e = 4 if case.get("prec") == "s" else 8
    if kind in ("posv", "potrf_potrs", "mixed"):
        n, m = case["n"], case["m"]
        by = e * (n * (n + 1) // 2 * (1 if kind == "mixed" else 2) + 2 * n * m) + 4
        fl = n ** 3 / 3 + n * n / 2 + n / 6 + 2 * m * n * n
        return {"bytes": batch * by, "flops": batch * fl}
    if kind in ("trsm", "trmm"):
        m, n = case["m"], case["n"]
        k = m if case["side"] == "L" else n
        return {"bytes": batch * e * (k * (k + 1) // 2 + 2 * m * n), "flops": batch * m * n * k}
    if kind == "syrk":
        m, k = case["m"], case["k"]
        return {"bytes": batch * e * (m * k + m * (m + 1)), "flops": batch * m * (m + 1) * k}
    if kind == "gemm_vbatch":
        m, n, k = (v.astype(np.float64) for v in _gemm_sizes(case))
        return {"bytes": float(e * (m * k + k * n + 2 * m * n).sum()),
                "flops": float(2 * (m * n * k).sum())}
    n = _vsizes(batch, case["nmin"], case["nmax"]).astype(np.float64)
    by = e * (n * (n + 1) / 2 * (1 if case["mixed"] else 2) + 2 * n) + 4
    return {"bytes": float(by.sum()),
            "flops": float((n ** 3 / 3 + n * n / 2 + n / 6 + 2 * n * n).sum())}


def _solve(a, bt):
    """Lower factor of a and the solution, for B^T columns bt (batch, n, m)."""
    lo = torch.linalg.cholesky(a)
    y = torch.linalg.solve_triangular(lo, bt, upper=False)
    return lo, torch.linalg.solve_triangular(lo.transpose(1, 2), y, upper=True)


def _first_bad(a):
    """1-based order of the first leading minor that is not positive definite."""
    n = a.shape[0]
    lo = np.zeros_like(a)
    for j in range(n):
        d = a[j, j] - lo[j, :j] @ lo[j, :j]
        if not d > 0:
            return j + 1
        lo[j:, j] = (a[j:, j] - lo[j:, :j] @ lo[j, :j]) / math.sqrt(d)
    return 0


def exact(case, seed):
    kind, p, batch = case["kind"], case.get("prec", "d"), case["batch"]
    g = _gen(seed)
    if kind in ("posv", "potrf_potrs", "mixed"):
        n, m = case["n"], case["m"]
        a = _spd(g, case.get("recipe", "shifted"), batch, n).to(DT[p]).double()
        b = _randn(g, batch, n, m).to(DT[p]).double()
        lo, x = _solve(a, b)
        info = torch.zeros(batch, dtype=torch.int32)
        if kind == "mixed":
            return {"x": x, "info": info}
        # [b, j, i]: L(i, j) for i >= j, the untouched upper part of A elsewhere
        return {"l": torch.triu(lo.transpose(1, 2)) + torch.tril(a, -1), "x": x, "info": info}
    if kind in ("trsm", "trmm"):
        m, n = case["m"], case["n"]
        k = m if case["side"] == "L" else n
        a = _tri(g, batch, k, case["uplo"], p).double().transpose(1, 2)  # A(i, j) at [b, i, j]
        b = _randn(g, batch, n, m).to(DT[p]).double().transpose(1, 2)
        op = a.transpose(1, 2) if case["trans"] == "T" else a
        up = (case["uplo"] == "U") != (case["trans"] == "T")
        if kind == "trmm":
            x = op @ b if case["side"] == "L" else b @ op
        else:
            x = torch.linalg.solve_triangular(op, b, upper=up, left=case["side"] == "L")
        return x.transpose(1, 2).contiguous()
    if kind == "syrk":
        m, k = case["m"], case["k"]
        a = (_randn(g, batch, k, m) if case["trans"] == "N" else _randn(g, batch, m, k)).to(DT[p]).double()
        c = _spd(g, "shifted", batch, m).to(DT[p]).double()
        # C is stored transposed; the product is symmetric
        new = c - (a.transpose(1, 2) @ a if case["trans"] == "N" else a @ a.transpose(1, 2))
        if case["uplo"] == "L":
            return torch.triu(new) + torch.tril(c, -1)
        return torch.tril(new) + torch.triu(c, 1)
    if kind == "gemm_vbatch":
        m, n, k = _gemm_sizes(case)
        sa, sb, sc = m * k, k * n, m * n
        a, b, c = (_randn(g, int(x.sum())).to(DT[p]).double() for x in (sa, sb, sc))
        oa, ob, oc = _offs(sa), _offs(sb), _offs(sc)
        out = c.clone()
        for i in range(batch):
            mi, ni, ki = int(m[i]), int(n[i]), int(k[i])
            ai = a[oa[i]:oa[i] + sa[i]].view((ki, mi) if case["transa"] == "N" else (mi, ki))
            bi = b[ob[i]:ob[i] + sb[i]].view((ni, ki) if case["transb"] == "N" else (ki, ni))
            ai = ai if case["transa"] == "N" else ai.t()   # op(A)^T, k x m
            bi = bi if case["transb"] == "N" else bi.t()   # op(B)^T, n x k
            out[oc[i]:oc[i] + sc[i]].view(ni, mi).addmm_(bi, ai, alpha=-1.0)
        return out
    ns, order, bad, offs, boffs, pool, b, _ = _vpool(case, seed)
    x = b.clone()
    info = np.zeros(batch, np.int32)
    k = 0
    while k < batch:
        n = int(ns[order[k]])
        e = k
        while e < batch and ns[order[e]] == n and not bad[order[e]]:
            e += 1
        if e == k:  # an indefinite system: B stays, info says where it failed
            i = order[k]
            info[i] = _first_bad(pool[offs[i]:offs[i] + n * n].view(n, n).cpu().numpy())
            k += 1
            continue
        o = int(offs[order[k]])
        at = torch.from_numpy(boffs[order[k:e]][:, None] + np.arange(n)).cuda()
        _, xs = _solve(pool[o:o + (e - k) * n * n].view(e - k, n, n), b[at][:, :, None])
        x[at] = xs[:, :, 0]
        k = e
    if case["mixed"]:
        return {"x": x, "info": torch.from_numpy(info)}
    return {"l": None, "x": x, "info": torch.from_numpy(info)}
