"""The single-matrix solve where it changes its way: factors with short and
long columns on both sides of the mean length, columns around the entries that
are loaded ahead, systems above the size whose vector is kept in shared
memory; and its division, pair by pair; against the host solve bit for bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from luspice_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solve(lib, n, f, q, b):
    import torch
    i32, f64 = torch.int32, torch.float64

    def dev(a, dtype):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")

    def p(t):
        return C.c_void_p(t.data_ptr())

    t = [dev(f[k], d) for k, d in (("Lp", i32), ("Li", i32), ("Lx", f64), ("Up", i32), ("Ui", i32), ("Ux", f64),
                                   ("pinv", i32))]
    dq, db, dx = dev(q, i32), dev(b, f64), torch.zeros(n, dtype=f64, device="cuda")
    wi, wd = torch.zeros(n, dtype=i32, device="cuda"), torch.zeros(2 * n, dtype=f64, device="cuda")
    assert lib.lusp_trisolve_par_launch(n, *map(p, t), p(dq), p(db), p(dx), p(wi), p(wd), None) == 0
    torch.cuda.synchronize()
    return dx.cpu().numpy()


def band(n, lower, upper, seed):
    r = np.random.default_rng(seed)
    return sp.diags([r.uniform(-1, 1, n - abs(o)) + (4.0 * (lower + upper) if o == 0 else 0.0)
                     for o in range(-lower, upper + 1)], range(-lower, upper + 1)).tocsc()


@pytest.mark.parametrize("n,lower,upper", [(700, 3, 60), (700, 60, 3), (500, 31, 32), (500, 32, 33), (500, 47, 47),
                                           (500, 48, 49), (900, 127, 128), (900, 128, 129), (900, 260, 300),
                                           (6001, 2, 3), (6001, 255, 256), (6001, 257, 258), (6100, 300, 40)])
def test_column_lengths_bitwise(gpu, lib, n, lower, upper):
    A = band(n, lower, upper, n + lower)
    q = np.arange(n, dtype=np.int32)
    f = api.pivot_factor(n, A.indptr, A.indices, A.data, q)
    b = np.random.default_rng(n).standard_normal(n)
    got, ref = solve(lib, n, f, q, b), O.lu_solve(f, q, b)
    assert np.array_equal(got.view(np.uint64), ref.view(np.uint64))


def divisions():
    """Dividends and divisors on both sides of the exponents +-400 between which
    the quotient is refined from a reciprocal, with mantissas at the ends of
    their range; zeros, subnormals, infinities and NaN."""
    r = np.random.default_rng(5)
    one = np.nextafter(1.0, 2.0)
    mant = np.array([1.0, one, 2.0 - 2.0 ** -52, 1.5, 4.0 / 3.0, np.nextafter(1.5, 0)])
    exps = [-1074, -1073, -1023, -1022, -1021, -402, -401, -400, -399, -1, 0, 1, 398, 399, 400, 401, 402, 1021, 1022, 1023]
    edge = np.concatenate([mant * 2.0 ** float(e) if e > -1023 else np.ldexp(mant, e) for e in exps]
                          + [np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324])])
    edge = np.concatenate([edge, -edge])
    a, d = np.meshgrid(edge, edge)
    wide = np.ldexp(r.uniform(1, 2, (2, 100000)), r.integers(-420, 420, (2, 100000)))
    near = np.ldexp(r.uniform(1, 2, (2, 100000)), r.integers(-3, 3, (2, 100000)))
    a, d = np.concatenate([a.ravel(), wide[0], near[0]]), np.concatenate([d.ravel(), wide[1], near[1]])
    keep = d != 1.0                  # a division that is skipped
    return a[keep] * r.choice([-1.0, 1.0], keep.sum()), d[keep]


@pytest.mark.parametrize("n", [5999, 6400])
def test_division_bitwise(gpu, lib, n):
    """x = b / U(k, k) of diagonal systems: the kernels' quotient is the
    correctly rounded one."""
    a, d = divisions()
    k = np.arange(n)
    f = {"Lp": np.arange(n + 1), "Li": k, "Lx": np.ones(n), "Up": np.arange(n + 1), "Ui": k, "pinv": k}
    with np.errstate(all="ignore"):
        for s in range(0, a.size, n):
            b, u = np.ones(n), np.full(n, 2.0)
            m = min(n, a.size - s)
            b[:m], u[:m] = a[s:s + m], d[s:s + m]
            got, exp = solve(lib, n, dict(f, Ux=u), k, b), b / u
            nan = np.isnan(exp)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.uint64), exp[~nan].view(np.uint64)), s
