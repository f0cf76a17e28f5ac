"""The lag-GEMM's work items at sizes where their length changes."""
import pytest

from seismic_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["laggemm", "laggemm16"])
@pytest.mark.parametrize("n,c,shift", [(1, 1, 30), (129, 1, 60), (300, 3, 128), (1500, 1, 200)])
def test_lag_items_of_every_size_agree(cuda_ok, form, n, c, shift):
    """The triangle's item size follows N; every pair against the FP32 spectra form at the lag form's tolerance."""
    import torch
    from seismic_gb300 import xcorr
    ev = torch.from_numpy(synth.family_catalog(n, c, 300, n_families=max(1, n // 40), seed=n)).cuda()
    a, b = xcorr.xcorr(ev, shift, form=form), xcorr.xcorr(ev, shift)
    tol = 1e-4 if form == "laggemm" else 2e-3
    assert (a.vals_pos - b.vals_pos).abs().max().item() < tol
    assert (a.vals_neg - b.vals_neg).abs().max().item() < tol
