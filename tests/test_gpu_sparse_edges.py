"""Compaction and histogram at the edges of their blocks, words and counter copies, against numpy."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _arrays(n, kept, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    vp = torch.rand(n, device="cuda", generator=g)
    vn = -torch.rand(n, device="cuda", generator=g)
    if n:
        vp[torch.rand(n, device="cuda", generator=g) >= kept] = 0.0
        vn[torch.rand(n, device="cuda", generator=g) >= kept] = 0.25 * vn[0]
        vp[-1], vn[-1] = 0.875, -1.0
    lp = torch.randint(-500, 500, (n,), device="cuda", generator=g, dtype=torch.int32)
    return vp, lp, vn, -lp


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("offset", [0, 1])  # 16-byte aligned arrays, and not
@pytest.mark.parametrize("n,kept", [(1, 1.0), (31, 1.0), (33, 0.5), (511, 0.1), (4095, 0.02), (4096, 1.0), (4097, 0.3),
                                    (70_001, 0.0), (5_000_003, 0.05)])
def test_compaction_edges(cuda_ok, n, kept, offset):
    import torch
    from seismic_gb300 import _lib
    lib = cuda_ok
    vp, lp, vn, ln = (torch.cat([x.new_zeros(offset), x])[offset:] for x in _arrays(n, kept, n))
    thr = 0.3
    full = lib.seismic_compact_workspace_bytes(n)
    counts_only = 16 * ((n + 4095) // 4096 + 1)
    a, b = np.flatnonzero(vp.cpu().numpy() > np.float32(thr)), np.flatnonzero(vn.cpu().numpy() < -np.float32(thr))
    for ws_bytes, split in ((full, False), (full, True), (counts_only, False), (counts_only, True)):
        for cap in (max(a.size, b.size, 1), max(1, a.size // 2)):
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
            counts = torch.zeros(2, dtype=torch.int64, device="cuda")
            out = [torch.full((cap,), -7, dtype=t, device="cuda")
                   for t in (torch.int64, torch.float32, torch.int32) * 2]
            args = [_ptr(vp), _ptr(lp), _ptr(vn), _ptr(ln), n, ctypes.c_float(thr)]
            s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            if split:
                _lib.check(lib.seismic_compact_pairs_device(*args, 0, *[None] * 6, _ptr(counts), _ptr(ws), ws_bytes, s))
                _lib.check(lib.seismic_compact_write_device(*args, cap, *map(_ptr, out), _ptr(ws), ws_bytes, s))
            else:
                _lib.check(lib.seismic_compact_pairs_device(*args, cap, *map(_ptr, out), _ptr(counts), _ptr(ws),
                                                            ws_bytes, s))
            assert counts.tolist() == [a.size, b.size]
            for idx, v, lag, (gi, gv, gl) in ((a, vp, lp, out[:3]), (b, vn, ln, out[3:])):
                m = min(cap, idx.size)
                np.testing.assert_array_equal(gi.cpu().numpy()[:m], idx[:m])
                np.testing.assert_array_equal(gv.cpu().numpy()[:m], v.cpu().numpy()[idx[:m]])
                np.testing.assert_array_equal(gl.cpu().numpy()[:m], lag.cpu().numpy()[idx[:m]])
                assert (gi.cpu().numpy()[m:] == -7).all()  # nothing past the capacity or the count


@pytest.mark.parametrize("nh", [1, 2, 19, 20, 190, 191, 1000, 4096, 4097, 20000])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 700_001])
def test_histogram_edges(cuda_ok, n, nh):
    from seismic_gb300 import sparse
    vp, _, vn, _ = _arrays(n, 0.7, n + nh)
    hmax, hmin = sparse.histogram(vp, vn, nh)
    delta = np.float32(1.0 / nh)
    for h, v in ((hmax, vp), (hmin, -vn)):
        v = v.cpu().numpy()
        b = np.minimum(np.where(v >= 1, nh - 1, (v / delta).astype(np.int32)), nh - 1)
        np.testing.assert_array_equal(h.cpu().numpy(), np.bincount(b, minlength=nh))
