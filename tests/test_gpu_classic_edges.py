"""The single-matrix kernels of lu_gpu_par.h where their work changes hands:
systems smaller than a bitmap word, columns long enough for all warps, rows
and columns without entries, capacities that run out, and solves around the
size up to which the vector is kept in shared memory; against the dense-scan
restatement and the host solve bit for bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from luspice_b200 import api, mna
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _t(torch, a, dtype):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _p(t):
    return C.c_void_p(t.data_ptr())


def factor(lib, A, q, lcap, ucap):
    import torch
    n = A.shape[0]
    t = {"Ap": _t(torch, A.indptr, torch.int32), "Ai": _t(torch, A.indices, torch.int32),
         "Ax": _t(torch, A.data, torch.float64), "dr": _t(torch, q, torch.int32)}
    for k, size, dt in (("Lp", n + 1, torch.int32), ("Up", n + 1, torch.int32), ("Li", lcap, torch.int32),
                        ("Ui", ucap, torch.int32), ("Lx", lcap, torch.float64), ("Ux", ucap, torch.float64),
                        ("pinv", n, torch.int32), ("xi", n + 2048, torch.int32), ("cnt", 3, torch.int32)):
        t[k] = torch.zeros(max(size, 1), dtype=dt, device="cuda")
    c = t["cnt"].data_ptr()
    rc = lib.lusp_lu_factor_par_launch(n, _p(t["Ap"]), _p(t["Ai"]), _p(t["Ax"]), _p(t["dr"]), _p(t["Lp"]), _p(t["Li"]),
                                       _p(t["Lx"]), lcap, _p(t["Up"]), _p(t["Ui"]), _p(t["Ux"]), ucap, _p(t["pinv"]),
                                       _p(t["xi"]), None, C.c_void_p(c), C.c_void_p(c + 4), C.c_void_p(c + 8), None)
    assert rc == 0
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in t.items()}


def matrix(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "dense":
        a = rng.uniform(-1.0, 1.0, (n, n)) + np.eye(n)
    elif kind == "diagonal":
        a = np.diag(rng.uniform(1.0, 2.0, n))
    else:       # "permuted": pivots off the diagonal, and ties
        a = np.zeros((n, n))
        a[rng.permutation(n), np.arange(n)] = 1.0
        a[rng.integers(0, n, 2 * n), rng.integers(0, n, 2 * n)] = rng.choice([-1.0, 1.0, 0.5], 2 * n)
    return sp.csc_matrix(a)


@pytest.mark.parametrize("kind,n", [("dense", n) for n in (1, 2, 3, 4, 5, 31, 32, 33, 65, 300, 600)]
                         + [("diagonal", 40), ("permuted", 97), ("permuted", 250)])
def test_factor_edges_bitwise(gpu, lib, kind, n):
    A = matrix(kind, n, n)
    q = np.arange(n, dtype=np.int32)
    exp = O.dense_factor(n, A.indptr, A.indices, A.data, q)
    cap = n * n + 64
    got = factor(lib, A, q, cap, cap)
    ln, un, sing = got["cnt"].tolist()
    assert sing == exp["status"]
    if sing != -1:
        return
    assert ln == exp["Lp"][-1] and un == exp["Up"][-1]
    for k in ("Lp", "Up", "pinv"):
        assert np.array_equal(got[k], exp[k]), k
    for k, cnt in (("Li", ln), ("Ui", un)):
        assert np.array_equal(got[k][:cnt], exp[k]), k
    for k, cnt in (("Lx", ln), ("Ux", un)):
        assert np.array_equal(got[k][:cnt].view(np.uint64), exp[k].view(np.uint64)), k


def test_factor_refusals(gpu, lib):
    """A singular column is named; capacities one short are refused."""
    m = mna.analog(200, 3)
    q = api.colamd(m.n, m.Ap, m.Ai)
    A = sp.csc_matrix((m.Ax, m.Ai, m.Ap), shape=(m.n, m.n))[:, q]
    A.sort_indices()
    exp = O.dense_factor(m.n, A.indptr, A.indices, A.data, q)
    ln, un = int(exp["Lp"][-1]), int(exp["Up"][-1])
    assert factor(lib, A, q, ln, un)["cnt"][2] == -1
    assert factor(lib, A, q, ln - 1, un)["cnt"][2] == -2
    assert factor(lib, A, q, ln, un - 1)["cnt"][2] == -2
    Z = A.copy()
    Z.data[Z.indptr[50]:Z.indptr[51]] = 0.0
    assert factor(lib, Z, q, ln, un)["cnt"][2] == 50


@pytest.mark.parametrize("n", [1, 31, 33, 64, 2500, 6000, 6001])
def test_solve_sizes_bitwise(gpu, lib, n):
    import torch
    if n < 100:
        A = matrix("dense", n, n)
        q = np.arange(n, dtype=np.int32)
        f = api.pivot_factor(n, A.indptr, A.indices, A.data, q)
    else:
        m = mna.analog(n, 4)
        q = api.colamd(m.n, m.Ap, m.Ai)
        f = api.pivot_factor(m.n, m.Ap, m.Ai, m.Ax, q)
    b = np.random.default_rng(n).standard_normal(n)
    ref = O.lu_solve(f, q, b)
    i32, f64 = torch.int32, torch.float64
    t = [_t(torch, f[k], d) for k, d in (("Lp", i32), ("Li", i32), ("Lx", f64), ("Up", i32), ("Ui", i32), ("Ux", f64),
                                         ("pinv", i32))]
    dq, db, dx = _t(torch, q, i32), _t(torch, b, f64), torch.zeros(n, dtype=f64, device="cuda")
    wi, wd = torch.zeros(n, dtype=i32, device="cuda"), torch.zeros(2 * n, dtype=f64, device="cuda")
    assert lib.lusp_trisolve_par_launch(n, *map(_p, t), _p(dq), _p(db), _p(dx), _p(wi), _p(wd), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(dx.cpu().numpy().view(np.uint64), ref.view(np.uint64))
