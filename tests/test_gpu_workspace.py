"""The workspace that refactorization (packed strict L) and solve (Krylov
vectors) share: a system's device memory, and factors and solutions when the
two alternate, with either of them the larger."""
import numpy as np
import pytest

from luspice_b200 import api, mna
from tests.helpers import TOL_REL, oracle_refactor, oracle_solution, rel_err

pytestmark = pytest.mark.gpu


def _al(b):
    return (b + 255) // 256 * 256


@pytest.mark.parametrize("prec,vs", [(api.MIXED, 4), (api.FP64, 8)])
def test_system_memory(gpu, prec, vs):
    """A batch takes the factor in the merged layout and by rows, the diagonal
    twice, A in SELL and the vectors: no further copy of the factor."""
    import torch
    m = mna.serving_class("grid", 2000, 3)
    P = api.Pattern.from_matrix(m, dense_tail=0)
    systems = 64
    api.Batch([P], prec=prec, ladder=0).close()         # loads the kernels
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    B = api.Batch([P] * systems, prec=prec, ladder=0)
    used = before - torch.cuda.mem_get_info()[0]
    B.close()
    n, i = P.n, P.info
    low, up = i["lnnz"] - n, i["unnz"] - n
    one = (_al(i["cap"] * vs + 64) + _al(low * vs + 64) + _al(up * vs + 64) + 2 * _al(n * vs + 64)
           + _al(14 * 2 * m.nnz) + 3 * 256                         # SELL copies (slices less than twice the entries)
           + _al((2 * 30 + 8) * n * 8) + 2 * _al(n * 8)           # Krylov vectors, scalings
           + 8 * m.nnz + 16 * n + 4096)                            # inputs, solution, descriptors
    assert used <= systems * one + (4 << 20), (used, systems * one)


@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
@pytest.mark.parametrize("krylov", [1, 30])
def test_refactor_and_solve_alternate(gpu, prec, krylov):
    m = mna.serving_class("grid", 1000, 5)
    P = api.Pattern.from_matrix(m, dense_tail=0)
    _, q = P.perm()
    vals = list(m.perturbed(3, seed=2))
    B = api.Batch([P, P], prec=prec, krylov=krylov, max_outer=30, ladder=0)
    ity = np.uint32 if prec == api.MIXED else np.uint64
    for a, b in ((0, 1), (2, 0)):
        B.upload([vals[a], vals[b]], [m.b, m.b])
        B.run(api.RUN_REFACTOR)
        exp = [oracle_refactor(m, P, vals[k], fp32=(prec == api.MIXED))[0] for k in (a, b)]
        for _ in range(2):
            for s in range(2):
                got = B.factor_values(s)
                assert np.array_equal(got.view(ity), exp[s].astype(got.dtype).view(ity))
            B.run(api.RUN_SOLVE)
            xs = B.split(B.download())
            for s, k in enumerate((a, b)):
                assert rel_err(xs[s], oracle_solution(m, vals[k], q=q)) <= TOL_REL
    B.close()
