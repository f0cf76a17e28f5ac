"""The lag-window scan and epilogue of the pair kernels at every transform size.

Window widths put the window's edges inside, between and outside the scan's
blocks of lags; the two-thread (P = 64), sub-warp, one-warp and multi-warp
groups finish their results in different ways.  Coefficients against the FP64
oracle, lags by the near-tie rule of tolerances.py; the histograms must be
exactly the reference's rule applied to the stored coefficients.
"""
import numpy as np
import pytest

from oracle import oracle as O
from seismic_gb300 import synth, xcorr
from tolerances import check_pairs

pytestmark = pytest.mark.gpu


def _bins(v, nh):
    """The reference's rule (Correlation_in_OMP/correlation_c.cpp:116-117): last bin for v >= 1, else int(v / delta) in
    float."""
    delta = np.float32(1.0 / nh)
    b = np.where(v >= 1, nh - 1, (v / delta).astype(np.int32))
    return np.bincount(np.minimum(b, nh - 1), minlength=nh)


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("padded", [64, 128, 256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("window", ["one", "narrow", "odd", "full"])
def test_scan_every_size(cuda_ok, monkeypatch, padded, window, direct):
    import torch
    if direct:
        monkeypatch.setenv("SEISMIC_PAIR_KERNEL", "direct")
    monkeypatch.setenv("SEISMIC_BLOCK_FORM", "off")
    shift = {"one": 1, "narrow": padded // 16 + 1, "odd": padded // 4 + 3, "full": padded // 2}[window]
    length = padded // 2 - (0 if window == "full" else 5)
    n, c, nh = 23, 1 + (padded // 64) % 2 * 2, 37
    ev = synth.family_catalog(n, c, length, n_families=3, seed=padded + shift)
    ev[5] = 0.0
    got = xcorr.xcorr(torch.from_numpy(ev).cuda(), shift, n_classes_hist=nh, padded_size=padded)
    vp, lp, vn, ln = (x.cpu().numpy() for x in (got.vals_pos, got.lags_pos, got.vals_neg, got.lags_neg))
    i, j = O.triu_pairs(n)
    r = O.fp64_xcorr(ev, shift, i, j, padded=padded)
    check_pairs((vp, lp, vn, ln), (r.val_pos, r.lag_pos, r.val_neg, r.lag_neg), r, 0.0, label=f"P={padded} {window}")
    live = (i != 5) & (j != 5)  # a pair with a zero event is not binned
    np.testing.assert_array_equal(got.max_hist.cpu().numpy(), _bins(vp[live], nh))
    np.testing.assert_array_equal(got.min_hist.cpu().numpy(), _bins(-vn[live], nh))


@pytest.mark.parametrize("nh", [1, 3, 10, 20, 100, 1000, 5000])
def test_bins_are_the_rounded_quotients(cuda_ok, nh):
    import torch
    ev = synth.ricker_catalog(150, 256, seed=nh)[:, 0]
    got = xcorr.xcorr(torch.from_numpy(ev).cuda(), 100, n_classes_hist=nh)
    np.testing.assert_array_equal(got.max_hist.cpu().numpy(), _bins(got.vals_pos.cpu().numpy(), nh))
    np.testing.assert_array_equal(got.min_hist.cpu().numpy(), _bins(-got.vals_neg.cpu().numpy(), nh))
