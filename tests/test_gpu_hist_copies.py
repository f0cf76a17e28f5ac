"""Standalone histograms at every number of counter copies (32, 16, 8, 4, 2, 1 and none), each copy filled, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh", [7, 190, 300, 500, 1000, 2000, 4096, 5000])
def test_copies_add_up(cuda_ok, nh):
    import torch
    from seismic_gb300 import sparse
    n = 300_001
    rng = np.random.default_rng(nh)
    vp, vn = rng.random(n, np.float32), -rng.random(n, np.float32)
    hists = sparse.histogram(torch.from_numpy(vp).cuda(), torch.from_numpy(vn).cuda(), nh)
    delta = np.float32(1.0 / nh)
    for h, v in zip(hists, (vp, -vn)):
        np.testing.assert_array_equal(h.cpu().numpy(), np.bincount((v / delta).astype(np.int32).clip(max=nh - 1), minlength=nh))
