"""SELL products on both sides of each rule that picks their kernel: slices and
long rows that fill the resident blocks, many and few long rows, short and very
long ones; against a host product."""
import numpy as np
import pytest
import scipy.sparse as sp

from luspice_b200 import api

pytestmark = pytest.mark.gpu


def check(rows, lengths, Cc, kind):
    """rows short rows of 1 to 3 entries, among them rows of `lengths`."""
    import torch
    rng = np.random.default_rng(rows + len(lengths))
    counts = rng.integers(1, 4, rows)
    at = rng.choice(rows, len(lengths), replace=False)
    counts[at] = lengths
    r = np.repeat(np.arange(rows), counts)
    c = rng.integers(0, rows, r.size)
    v = np.ldexp(rng.uniform(1.0, 2.0, r.size), rng.integers(-2, 3, r.size)) * rng.choice([-1.0, 1.0], r.size)
    rowptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    if kind == "fp32":
        v = v.astype(np.float32).astype(np.float64)
    x = rng.standard_normal(rows)
    S = api.Sell(rows, rowptr, c.astype(np.int32), v, Cc, 256, kind)
    dx = torch.as_tensor(x, device="cuda")
    dy = torch.full((rows,), np.nan, dtype=torch.float64, device="cuda")
    S.spmv(dx.data_ptr(), dy.data_ptr())
    torch.cuda.synchronize()
    ref, scale = np.add.reduceat(v * x[c], rowptr[:-1]), np.add.reduceat(np.abs(v * x[c]), rowptr[:-1])
    # fp64 sums of at most n products on both sides: 2 n 2^-53.
    tol = 2 * (counts.max() + 8) * 2.0 ** -53 * scale
    assert np.all(np.abs(dy.cpu().numpy() - ref) <= tol)


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kind", ["fp64", "fp32"])
@pytest.mark.parametrize("Cc", [8, 16, 32])
@pytest.mark.parametrize("more", [0, 1])
def test_slices_fill_the_resident_blocks(gpu, Cc, kind, more):
    """4 blocks of 8 warps per SM, and one slice more."""
    check(32 * sms() * Cc + more, [], Cc, kind)


@pytest.mark.parametrize("kind", ["fp64", "fp32"])
@pytest.mark.parametrize("more", [0, 1])
def test_long_rows_fill_the_resident_blocks(gpu, kind, more):
    """Slices in 2 blocks per SM, long rows in the other 2, and one more."""
    check(16 * sms() * 32, [300] * (2 * sms() + more), 32, kind)


@pytest.mark.parametrize("kind", ["fp64", "fp32"])
@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("length", [257, 288, 352, 383, 384, 385, 641, 767, 768, 800])
def test_rows_by_block_and_by_warp(gpu, length, many, kind):
    """8 rows per SM, and more of them in a matrix whose mean keeps them long."""
    n = 8 * sms() + (1 if many else 0)
    check(60 * n, [length] * n, 32, kind)


@pytest.mark.parametrize("kind", ["fp64", "fp32"])
@pytest.mark.parametrize("rows,nlong,length", [(60000, 600, 4096), (60000, 600, 4095), (60000, 600, 9000),
                                               (1500000, 4, 9000)])
def test_very_long_rows(gpu, rows, nlong, length, kind):
    check(rows, [length] * nlong, 32, kind)
