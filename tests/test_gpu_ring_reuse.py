"""The staged pair kernel where every CTA walks many items, so that ring slots, their phases and (past 32 items a CTA) the ring of
decoded items come round again: slots of 2, 4 and 8 chunks and, on plain transforms, the direct form give the same bits."""
import pytest

from seismic_gb300 import synth, xcorr

pytestmark = pytest.mark.gpu

FIELDS = ("vals_pos", "lags_pos", "vals_neg", "lags_neg", "max_hist", "min_hist")


@pytest.mark.parametrize("n,c,length,shift,form,plain", [
    (300, 1, 512, 512, "fp32", True), (811, 1, 512, 512, "fp32", True),       # P = 1024, one row: 11 and 80 items a CTA
    (301, 1, 1024, 1024, "fp32", True), (431, 1, 1024, 1024, "fp32", True),   # P = 2048, one row: two slots; 23 and 46 items
    (301, 1, 1024, 128, "fp32", False), (900, 1, 1024, 128, "fp16", False),   # overlap-save, Q = 512 x 4
    (303, 3, 512, 512, "fp32", True), (251, 3, 1000, 250, "fp32", False),     # three channels; Q = 1024 x 2 frames of them
    (401, 1, 1024, 1000, "fp16", True), (700, 1, 256, 256, "bf16", True),     # half types at P = 2048 and 512
    (149, 3, 2048, 2048, "fp32", True)])                                      # P = 4096: 2 against 4 chunks
def test_slots_and_items_come_round(cuda_ok, monkeypatch, n, c, length, shift, form, plain):
    import torch
    ev = torch.from_numpy(synth.family_catalog(n, c, length, n_families=max(1, n // 16), seed=n)).cuda()
    got = {}
    for ru in ("2", "4", "8"):
        monkeypatch.setenv("SEISMIC_STAGED_RU", ru)
        got[ru] = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
    monkeypatch.delenv("SEISMIC_STAGED_RU")
    monkeypatch.setenv("SEISMIC_STAGED_WARPS", "12")
    got["12 warps"] = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
    monkeypatch.delenv("SEISMIC_STAGED_WARPS")
    if plain:
        monkeypatch.setenv("SEISMIC_PAIR_KERNEL", "direct")
        got["direct"] = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
        monkeypatch.delenv("SEISMIC_PAIR_KERNEL")
    rule = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
    for k, r in got.items():
        for f in FIELDS:
            assert torch.equal(getattr(r, f), getattr(rule, f)), (k, f)
