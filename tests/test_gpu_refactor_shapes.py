"""How the systems of a batch of medium circuits share the GPU in the
refactorization, on both sides of the batch size where it changes, and the
factor's bits there."""
import numpy as np
import pytest

from luspice_b200 import api, mna
from tests.helpers import oracle_refactor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [api.MIXED, api.FP64])
def test_medium_batches(gpu, prec):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = mna.serving_class("grid", 1000, 5)
    P = api.Pattern.from_matrix(m)
    assert P.info["gathered"] > 1 << 17
    vals = list(m.perturbed(2, seed=2))
    exp = [oracle_refactor(m, P, v, fp32=(prec == api.MIXED))[0] for v in vals]
    ity = np.uint32 if prec == api.MIXED else np.uint64
    # Six CTAs of 256 threads per system, four on an SM; five; four.
    for systems, spread in ((4 * sms // 6, 6), (4 * sms // 6 + 1, 0), (sms, 0)):
        B = api.Batch([P] * systems, prec=prec, krylov=4, ladder=0)
        B.upload(np.concatenate([vals[s % 2] for s in range(systems)]), np.tile(m.b, systems))
        B.run(api.RUN_REFACTOR)
        shape = B.launch_shape()
        assert (shape["refactor_spread"], shape["refactor_block"]) == (spread, 256 if spread else 768), systems
        for s in (0, systems - 1):
            got = B.factor_values(s)
            assert np.array_equal(got.view(ity), exp[s % 2].astype(got.dtype).view(ity)), (systems, s)
        B.close()
