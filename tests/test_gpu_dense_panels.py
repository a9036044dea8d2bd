"""Dense trailing block at the edges of its tiling: block sizes around the
32-column panels, the CTA's row count and the largest block, on a 2-CTA
cluster and on a lone CTA, against the host restatement bit for bit, and the
pivot statistics against the factorization without a dense block (value sets
with multipliers above 1, and scaled so far that the division leaves the range
of its refinement)."""
import numpy as np
import pytest

from luspice_b200 import api, mna
from tests.helpers import oracle_refactor

pytestmark = pytest.mark.gpu

STATS = ("min_abs_pivot", "min_pivot_ratio", "max_abs_u", "singular_col")


def _bits(a):
    return a.view(np.uint32 if a.dtype == np.float32 else np.uint64)


def _factors(m, vals, tail, copies, prec):
    """Factor values and statistics of value sets vals, each in a batch of
    `copies` systems (few: a 2-CTA cluster per system; many: a lone CTA)."""
    P = api.Pattern.from_matrix(m, dense_tail=tail)
    assert P.info["dense_tail"] == tail
    nsys = max(copies, len(vals))
    B = api.Batch([P] * nsys, prec=prec)
    B.upload([vals[s % len(vals)] for s in range(nsys)], [m.b] * nsys)
    B.run(api.RUN_REFACTOR)
    picks = range(nsys - len(vals), nsys)
    out = {s % len(vals): (B.factor_values(s), B.stats()[s]) for s in picks}
    shape = B.launch_shape()
    B.close()
    return P, out, shape


@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
@pytest.mark.parametrize("copies,cluster", [(2, 2), (150, 1)])
@pytest.mark.parametrize("tail", [1, 31, 32, 33, 64, 95, 129, 256])
def test_panel_edges_bitwise(gpu, tail, copies, cluster, prec):
    m = mna.analog(300, 9)
    vals = list(m.perturbed(2, seed=tail, sigma=1.0)) + [m.Ax * 1e-200]
    P, out, shape = _factors(m, vals, tail, copies if copies > 2 else 3, prec)
    assert shape["dense_cluster"] == cluster
    _, ref, _ = _factors(m, vals, 0, 3, prec)
    for s, v in enumerate(vals):
        exp, _ = oracle_refactor(m, P, v, fp32=(prec == api.MIXED))
        got, st = out[s]
        assert np.array_equal(_bits(got), _bits(exp.astype(got.dtype))), (tail, s)
        for k in STATS:
            assert st[k] == ref[s][1][k], (tail, s, k)


@pytest.mark.parametrize("tail", [320, 511, 513, 768])
def test_large_blocks_bitwise(gpu, tail):
    """Rows past the CTA's threads, and the largest block (one copy group in
    flight per warp)."""
    m = mna.analog(989, 42)
    vals = list(m.perturbed(2, seed=tail))
    P, out, _ = _factors(m, vals, tail, 2, api.FP64)
    for s, v in enumerate(vals):
        exp, bad = oracle_refactor(m, P, v, fp32=False)
        assert bad < 0
        assert np.array_equal(_bits(out[s][0]), _bits(exp)), (tail, s)
