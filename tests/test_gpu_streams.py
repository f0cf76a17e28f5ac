"""xcorr(stream=...): the whole call runs on the stream it is given, whatever torch's current stream is doing."""
import pytest

from seismic_gb300 import synth, xcorr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("nh", [0, 20])
def test_side_stream_does_not_wait_for_the_current_one(cuda_ok, strided, nh):
    """The current stream sleeps; the call on a side stream is complete, its histograms included, before that ends."""
    import torch
    ev = torch.from_numpy(synth.family_catalog(60, 1, 256, n_families=3, seed=1)).cuda()
    if strided:
        ev = torch.stack((ev, -ev), -1)[..., 0]
    side = torch.cuda.Stream()
    xcorr.xcorr(ev, 100, n_classes_hist=nh, stream=side)  # first-call set-up
    want = xcorr.xcorr(ev, 100, n_classes_hist=nh)
    names = ("vals_pos", "lags_pos", "vals_neg", "lags_neg", "max_hist", "min_hist")
    want = [getattr(want, k).cpu() for k in names]
    torch.cuda.synchronize()
    torch.cuda._sleep(600_000_000)  # about 0.3 s of the current stream
    got = xcorr.xcorr(ev, 100, n_classes_hist=nh, stream=side)
    side.synchronize()
    with torch.cuda.stream(side):
        got = [getattr(got, k).cpu() for k in names]
    assert not torch.cuda.current_stream().query()
    for k, g, w in zip(names, got, want):
        assert torch.equal(g, w), k
    torch.cuda.synchronize()
