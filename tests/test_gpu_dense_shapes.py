"""Dense trailing blocks on lone CTAs: the CTA size for the systems per SM, and
the factor's bits with every size, up to the largest block (rows past the
CTA's threads, one copy group in flight per warp)."""
import numpy as np
import pytest

from luspice_b200 import api, mna
from tests.helpers import oracle_refactor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
@pytest.mark.parametrize("tail,per_sm,threads", [
    (33, 1, 512), (96, 1, 512), (128, 1, 512), (256, 1, 512), (320, 1, 512), (513, 1, 512), (768, 1, 512),
    (33, 2, 256), (128, 2, 256), (129, 2, 256), (256, 2, 256), (257, 2, 512),
    (33, 3, 128), (128, 3, 128), (129, 3, 256), (256, 3, 256), (320, 3, 512)])
def test_lone_cta_sizes_bitwise(gpu, tail, per_sm, threads, prec):
    import torch
    m = mna.analog(max(300, tail + 20), 9)
    P = api.Pattern.from_matrix(m, dense_tail=tail)
    assert P.info["dense_tail"] == tail
    systems = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    vals = list(m.perturbed(2, seed=tail))
    B = api.Batch([P] * systems, prec=prec, krylov=4, ladder=0)
    B.upload(np.concatenate([vals[s % 2] for s in range(systems)]), np.tile(m.b, systems))
    B.run(api.RUN_REFACTOR)
    shape = B.launch_shape()
    assert (shape["dense_cluster"], shape["dense_block"]) == (1, threads)
    ity = np.uint32 if prec == api.MIXED else np.uint64
    for s in (0, systems - 1):
        exp, _ = oracle_refactor(m, P, vals[s % 2], fp32=(prec == api.MIXED))
        got = B.factor_values(s)
        assert np.array_equal(got.view(ity), exp.astype(got.dtype).view(ity)), s
    B.close()
