"""The single-matrix factorization on patterns other than circuits: columns
whose updates are shared by all warps, columns that touch more rows than the
row list holds (the bitmap is walked instead), rows and columns without
entries, and input columns with repeated rows; against the dense-scan
restatement bit for bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from tests.test_gpu_classic_edges import _p, factor

pytestmark = pytest.mark.gpu


def check(lib, A):
    n = A.shape[0]
    q = np.arange(n, dtype=np.int32)
    exp = O.dense_factor(n, A.indptr, A.indices, A.data, q)
    ln, un = (int(exp["Lp"][-1]), int(exp["Up"][-1])) if exp["status"] == -1 else (n * n, n * n)
    got = factor(lib, A, q, ln, un)
    assert got["cnt"][2] == exp["status"]
    if exp["status"] != -1:
        return exp
    assert got["cnt"].tolist()[:2] == [ln, un]
    for k in ("Lp", "Up", "pinv", "Li", "Ui"):
        assert np.array_equal(got[k], exp[k]), k
    for k in ("Lx", "Ux"):
        assert np.array_equal(got[k].view(np.uint64), exp[k].view(np.uint64)), k
    return exp


@pytest.mark.parametrize("bandwidth", [16, 31, 32, 33, 34, 64, 257, 300])
def test_update_lengths(gpu, lib, bandwidth):
    n = 2 * bandwidth + 70
    r = np.random.default_rng(bandwidth)
    A = sp.diags([r.uniform(-1, 1, n - abs(o)) for o in range(-bandwidth, bandwidth + 1)],
                 range(-bandwidth, bandwidth + 1)).tocsc()
    check(lib, A)


def arrow(n, full, seed):
    """A diagonal, the columns `full` without a zero, and a few scattered
    entries."""
    r = np.random.default_rng(seed)
    a = sp.random(n, n, 2.0 / n, random_state=seed, data_rvs=lambda k: r.uniform(-1, 1, k)).tolil()
    a.setdiag(r.uniform(1.0, 2.0, n))
    for c in full:
        a[:, c] = r.uniform(-1.0, 1.0, (n, 1))
    return a.tocsc()


@pytest.mark.parametrize("full", [[0], [600], [1249], [3, 600, 601, 1249]])
def test_more_rows_than_the_list_holds(gpu, lib, full):
    n = 1250
    A = arrow(n, full, len(full))
    assert np.diff(A.indptr).max() == n > (12 * n + 256 - 10 * n - 8 * ((n + 31) // 32)) // 2
    exp = check(lib, A)
    ln, un = int(exp["Lp"][-1]), int(exp["Up"][-1])
    q = np.arange(n, dtype=np.int32)
    assert factor(lib, A, q, ln - 1, un)["cnt"][2] == -2
    assert factor(lib, A, q, ln, un - 1)["cnt"][2] == -2


@pytest.mark.parametrize("n,at", [(70, 0), (70, 33), (70, 69), (1250, 640)])
def test_empty_rows_and_columns(gpu, lib, n, at):
    A = arrow(n, [5], 3).tolil()
    B = A.copy()
    B[:, at] = 0.0
    B = B.tocsc()
    B.eliminate_zeros()
    assert check(lib, B)["status"] == at
    A[at, :] = 0.0
    A = A.tocsc()
    A.eliminate_zeros()
    assert check(lib, A)["status"] >= 0


@pytest.mark.parametrize("n", [20, 40, 150])
def test_repeated_rows_take_the_last(gpu, lib, n):
    """Columns of up to 4 n entries in no order, rows repeated inside a group
    of 32 entries and across groups: the last entry of a row counts."""
    r = np.random.default_rng(n)
    ptr, rows, vals = [0], [], []
    dense = np.zeros((n, n))
    for c in range(n):
        k = r.choice([n, 31, 33, 64, 4 * n])
        i = np.concatenate([r.integers(0, n, k), [c]])
        v = np.concatenate([r.uniform(-1, 1, k), [float(n)]])
        rows.append(i)
        vals.append(v)
        ptr.append(ptr[-1] + i.size)
        dense[i, c] = v             # in order: the last one stays
    A = sp.csc_matrix((n, n))
    A.indptr, A.indices, A.data = np.array(ptr, np.int32), np.concatenate(rows).astype(np.int32), np.concatenate(vals)
    D = sp.csc_matrix(dense)
    q = np.arange(n, dtype=np.int32)
    cap = n * n + n
    exp = check(lib, D)
    got = factor(lib, A, q, cap, cap)
    assert got["cnt"][2] == -1
    for k, m in (("Lp", None), ("Up", None), ("pinv", None), ("Li", exp["Li"].size), ("Ui", exp["Ui"].size)):
        assert np.array_equal(got[k][:m], exp[k]), k
    for k in ("Lx", "Ux"):
        assert np.array_equal(got[k][:exp[k].size].view(np.uint64), exp[k].view(np.uint64)), k


def test_input_columns_cost_their_length(gpu, lib):
    """Dense lower triangles have no updates, only input: four times the columns
    and rows are 16 times the entries, and no more than 32 times the time (a
    search for repeated rows over the rest of a column would make it 64)."""
    import torch
    times = []
    for n in (300, 1200):
        A = sp.csc_matrix(np.tril(np.random.default_rng(n).uniform(-1, 1, (n, n))) + n * np.eye(n))
        q, cap = np.arange(n, dtype=np.int32), n * n
        t = {k: torch.as_tensor(v, device="cuda") for k, v in (("Ap", A.indptr), ("Ai", A.indices), ("Ax", A.data), ("q", q))}
        for k, size, dt in (("Lp", n + 1, torch.int32), ("Up", n + 1, torch.int32), ("Li", cap, torch.int32),
                            ("Ui", cap, torch.int32), ("Lx", cap, torch.float64), ("Ux", cap, torch.float64),
                            ("pinv", n, torch.int32), ("xi", n + 2048, torch.int32), ("cnt", 3, torch.int32)):
            t[k] = torch.zeros(size, dtype=dt, device="cuda")
        stream, c, best = torch.cuda.current_stream(), t["cnt"].data_ptr(), np.inf
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            assert lib.lusp_lu_factor_par_launch(
                n, _p(t["Ap"]), _p(t["Ai"]), _p(t["Ax"]), _p(t["q"]), _p(t["Lp"]), _p(t["Li"]), _p(t["Lx"]), cap,
                _p(t["Up"]), _p(t["Ui"]), _p(t["Ux"]), cap, _p(t["pinv"]), _p(t["xi"]), None, C.c_void_p(c),
                C.c_void_p(c + 4), C.c_void_p(c + 8), C.c_void_p(stream.cuda_stream)) == 0
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        assert t["cnt"].tolist() == [n * (n + 1) // 2, n, -1]
        times.append(best)
    assert times[1] <= 32 * times[0], times
