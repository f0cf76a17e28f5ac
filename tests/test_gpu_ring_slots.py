"""The staged pair kernel's ring slots of 2, 4 and 8 chunks give the same bits, at sizes with ragged last tiles, with one and
several spectrum rows, full and half-precision spectra, and where the longest slot does not fit."""
import pytest

from seismic_gb300 import synth, xcorr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,length,shift,form", [
    (1, 1, 256, 256, "fp32"), (31, 1, 1024, 128, "fp32"), (97, 3, 256, 200, "fp16"), (61, 1, 512, 512, "fp32"),
    (64, 3, 1000, 250, "fp32"), (63, 3, 1000, 250, "bf16"), (45, 1, 1024, 1024, "fp32"), (33, 3, 900, 1000, "fp32"),
    (47, 1, 1024, 1000, "fp16"), (19, 3, 2048, 2048, "fp32"), (13, 1, 2000, 1800, "bf16")])
def test_ring_slots_agree_bitwise(cuda_ok, monkeypatch, n, c, length, shift, form):
    import torch
    ev = torch.from_numpy(synth.family_catalog(n, c, length, n_families=max(1, n // 16), seed=n)).cuda()
    got = {}
    for ru in ("2", "4", "8"):
        monkeypatch.setenv("SEISMIC_STAGED_RU", ru)
        got[ru] = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
    monkeypatch.delenv("SEISMIC_STAGED_RU")
    got["rule"] = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
    for k in ("2", "4", "8"):
        for f in ("vals_pos", "lags_pos", "vals_neg", "lags_neg", "max_hist", "min_hist"):
            assert torch.equal(getattr(got[k], f), getattr(got["rule"], f)), (k, f)
