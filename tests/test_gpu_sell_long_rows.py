"""SELL rows kept out of the slices (a block per row) at the edges of a block's
rounds: row lengths around 256, 768 and 1024 entries, every value storage that
fits, against a host product."""
import numpy as np
import pytest
import scipy.sparse as sp

from luspice_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("length", [257, 512, 767, 768, 769, 1023, 1024, 1025, 1793, 3000])
def test_long_row_lengths(gpu, length, kind):
    import torch
    n = 3100
    rng = np.random.default_rng(length)
    rows = [0, 1500, n - 1]
    r = np.concatenate([np.arange(n)] + [np.full(length - 1, i) for i in rows])
    c = np.concatenate([np.arange(n)] + [rng.choice(np.delete(np.arange(n), i), length - 1, replace=False) for i in rows])
    A = sp.csr_matrix((rng.uniform(0.5, 2.0, r.size) * rng.choice([-1.0, 1.0], r.size), (r, c)), shape=(n, n))
    A.sort_indices()
    assert A.indptr[1] - A.indptr[0] == length
    x = rng.standard_normal(n)
    S = api.Sell(n, A.indptr, A.indices, A.data, 32, 256, kind)
    dx = torch.as_tensor(x, device="cuda")
    dy = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    S.spmv(dx.data_ptr(), dy.data_ptr())
    torch.cuda.synchronize()
    v = A.data.astype(np.float32).astype(np.float64) if kind == "fp32" else A.data
    ref = sp.csr_matrix((v, A.indices, A.indptr), shape=A.shape) @ x
    scale = np.abs(A) @ np.abs(x)
    # fp64 sums of at most `length` products: length * 2^-53; fp16 storage: 2^-11 an entry.
    tol = 2.0 ** -11 + 1e-9 if kind == "fp16" else (length + 8) * 2.0 ** -53
    assert np.all(np.abs(dy.cpu().numpy() - ref) <= tol * scale)


@pytest.mark.parametrize("Cc", [8, 16, 32])
@pytest.mark.parametrize("n", [1, 31, 33, 189440, 189473])
def test_slice_loads(gpu, n, Cc):
    """Short and long slices on both sides of the size up to which a slice's
    entries are requested together."""
    import torch
    rng = np.random.default_rng(n)
    counts = rng.integers(1, 20, n) if n < 1000 else rng.integers(1, 8, n)
    counts = np.minimum(counts, n)
    r = np.repeat(np.arange(n), counts)
    c = (r + rng.integers(0, max(1, n // 3), r.size)) % n
    A = sp.csr_matrix((rng.standard_normal(r.size), (r, c)), shape=(n, n))
    A.sort_indices()
    x = rng.standard_normal(n)
    S = api.Sell(n, A.indptr, A.indices, A.data, Cc, 256, "fp64")
    dx = torch.as_tensor(x, device="cuda")
    dy = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    S.spmv(dx.data_ptr(), dy.data_ptr())
    torch.cuda.synchronize()
    assert np.all(np.abs(dy.cpu().numpy() - A @ x) <= 40 * 2.0 ** -53 * (abs(A) @ np.abs(x)) + 1e-300)
