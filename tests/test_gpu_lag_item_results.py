"""The lag-GEMM's items of every length give the same bits: a catalog's pairs do not depend on how many events follow (its length
picks the triangle's items), a request's on the queries an item takes; lags and histograms included."""
import numpy as np
import pytest

from seismic_gb300 import synth, xcorr

pytestmark = pytest.mark.gpu

FIELDS = ("vals_pos", "lags_pos", "vals_neg", "lags_neg")


def _bins(v, nh):
    """The reference's rule (Correlation_in_OMP/correlation_c.cpp:116-117)."""
    b = np.where(v >= 1, nh - 1, (v / np.float32(1.0 / nh)).astype(np.int32))
    return np.bincount(np.minimum(b, nh - 1), minlength=nh)


@pytest.mark.parametrize("form", ["laggemm", "laggemm16"])
@pytest.mark.parametrize("c,length,shift", [(1, 300, 128), (3, 128, 30), (1, 1000, 200), (1, 64, 16)])
def test_a_prefix_of_the_catalog_gives_the_same_pairs(cuda_ok, form, c, length, shift):
    import torch
    n, nh = 2600, 20
    ev = torch.from_numpy(synth.family_catalog(n, c, length, n_families=60, seed=length)).cuda()
    whole = xcorr.xcorr(ev, shift, form=form)
    for m in (1, 2, 129, 300, 601, 1500):
        part = xcorr.xcorr(ev[:m], shift, form=form, n_classes_hist=nh)
        i, j = np.triu_indices(m)
        at = torch.from_numpy(xcorr.packed_index(i, j, n)).cuda()
        for f in FIELDS:
            assert torch.equal(getattr(part, f), getattr(whole, f)[at]), (m, f)
        np.testing.assert_array_equal(part.max_hist.cpu().numpy(), _bins(part.vals_pos.cpu().numpy(), nh))
        np.testing.assert_array_equal(part.min_hist.cpu().numpy(), _bins(-part.vals_neg.cpu().numpy(), nh))


@pytest.mark.parametrize("form", ["laggemm", "laggemm16"])
@pytest.mark.parametrize("c,length,shift", [(1, 300, 60), (3, 512, 256)])  # two events a pass, and one
def test_a_request_does_not_depend_on_its_items(cuda_ok, monkeypatch, form, c, length, shift):
    from seismic_gb300.serving import Server
    cat = synth.family_catalog(1300, c, length, n_families=20, seed=4)
    srv = Server(cat, shift=shift, form=form, n_slots=1, max_query_events=64, topk=8)
    for nq in (1, 2, 3, 5, 64):
        q = synth.family_catalog(nq, c, length, n_families=2, seed=nq)
        for subset in ((0, 1300), (100, 300), (37, 38)):
            want = srv.wait(srv.submit(q, subset=subset))
            for jc in ("1", "2", "4", "8"):
                monkeypatch.setenv("SEISMIC_LAG_RECT_JC", jc)
                got = srv.wait(srv.submit(q, subset=subset))
                for f in (*FIELDS, "topk_vals", "topk_index"):
                    np.testing.assert_array_equal(getattr(got, f), getattr(want, f))
            monkeypatch.delenv("SEISMIC_LAG_RECT_JC")
    srv.close()
