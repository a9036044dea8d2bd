"""Update segments of the refactorization (consecutive columns of one
supernode) at the edges of a warp: supernodes around 32 columns, updates of
one, two and more 32-row chunks, more than 32 segments in a column, and work
vectors that spill, under every way the columns of a system are shared,
against the host restatement bit for bit."""
import numpy as np
import pytest

from luspice_b200 import api
from tests.helpers import oracle_refactor

pytestmark = pytest.mark.gpu


class Matrix:
    """A CSC matrix with the fields the helpers read."""

    def __init__(self, a, seed):
        n = a.shape[0]
        cols, rows = np.nonzero(a.T)
        self.n, self.nnz = n, rows.size
        self.Ai = rows.astype(np.int32)
        self.Ap = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32)
        self.Ax = a.T[cols, rows].copy()
        self.b = np.random.default_rng(seed).uniform(-1, 1, n)


def dense(n, seed):
    """One supernode of n columns."""
    a = np.random.default_rng(seed).uniform(-1.0, 1.0, (n, n))
    return Matrix(a + n * np.eye(n), seed)


def blocks(widths, border, seed):
    """Independent dense blocks and a dense border of rows and columns: a
    border column has a segment per block (and one for the border)."""
    rng = np.random.default_rng(seed)
    n = sum(widths) + border
    a = np.zeros((n, n))
    o = 0
    for w in widths:
        a[o:o + w, o:o + w] = rng.uniform(-1.0, 1.0, (w, w))
        o += w
    a[o:, :] = rng.uniform(-1.0, 1.0, (border, n))
    a[:, o:] = rng.uniform(-1.0, 1.0, (n, border))
    return Matrix(a + 4 * n * np.eye(n), seed)


def check(m, prec, systems=2, zeros=False, **opts):
    q = np.arange(m.n, dtype=np.int32)
    P = api.Pattern.from_matrix(m, q=q, dense_tail=0)
    rng = np.random.default_rng(m.n)
    vals = [m.Ax * np.exp(0.1 * rng.standard_normal(m.nnz)) for _ in range(systems)]
    if zeros:       # exact zeros in U: their columns apply nothing
        cols = np.repeat(np.arange(m.n), np.diff(m.Ap))
        vals[0] = np.where((m.Ai < m.n // 2) & (cols > m.Ai) & (rng.random(m.nnz) < 0.5), 0.0, vals[0])
    B = api.Batch([P] * systems, prec=prec, **opts)
    B.upload(vals, [m.b] * systems)
    B.run(api.RUN_REFACTOR)
    for s in (0, systems - 1):
        exp, _ = oracle_refactor(m, P, vals[s], fp32=(prec == api.MIXED))
        got = B.factor_values(s)
        ity = np.uint32 if prec == api.MIXED else np.uint64
        assert np.array_equal(got.view(ity), exp.astype(got.dtype).view(ity)), (m.n, s, opts)
    shape = B.launch_shape()
    B.close()
    return shape


SHAPES = [dict(refactor_cluster=1), dict(refactor_cluster=2), dict(refactor_spread=3)]


@pytest.mark.parametrize("opts", SHAPES)
@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 34, 64, 65, 66, 97, 130])
def test_one_supernode(gpu, n, prec, opts):
    check(dense(n, n), prec, zeros=n > 30, **opts)


@pytest.mark.parametrize("opts", SHAPES)
@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
@pytest.mark.parametrize("widths,border", [([1] * 40, 5), ([2, 5, 1, 33, 3, 40, 1], 12), ([4] * 70, 40)])
def test_many_segments(gpu, widths, border, prec, opts):
    check(blocks(widths, border, 3), prec, **opts)


@pytest.mark.parametrize("opts", [dict(refactor_threads=512, refactor_cluster=1), dict(refactor_mode=1)])
def test_spilled_and_searched_columns(gpu, opts):
    """Columns longer than a warp's work area (global memory), and the path
    that searches a column's rows."""
    check(blocks([5, 1, 40] * 30, 70, 5), api.FP64, **opts)


def test_shapes_are_taken(gpu):
    m = blocks([2, 5, 1, 33], 12, 3)
    assert check(m, api.MIXED, refactor_cluster=2)["refactor_cluster"] == 2
    assert check(m, api.MIXED, refactor_spread=3)["refactor_spread"] == 3
    assert check(m, api.MIXED, systems=160)["refactor_cluster"] == 1
