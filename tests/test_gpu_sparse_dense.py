"""Compaction of chunks (512 pairs, 1024 with both sides) that keep few, about half or all of their pairs, where the write pass
changes from finding each round's pairs to going word by word; against numpy, from every kind of workspace."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [0, 1, 31, 33, 64, 255, 511, 512, 513, 900, 1023, 1024])
@pytest.mark.parametrize("chunks", [1, 8, 9, 700])
@pytest.mark.parametrize("with_words", [True, False])
def test_chunks_that_keep(cuda_ok, kept, chunks, with_words):
    import torch
    from seismic_gb300 import _lib
    lib = cuda_ok
    rng = np.random.default_rng(kept * 1000 + chunks)
    n = 512 * chunks - (37 if kept < 900 and chunks > 1 else 0)  # a ragged last chunk
    mask = np.zeros((chunks, 1024), bool)
    for m in mask:
        m[rng.permutation(1024)[:kept]] = True
    pos, neg = mask[:, :512].ravel()[:n], mask[:, 512:].ravel()[:n]
    vp = np.where(pos, rng.uniform(0.5, 1, n), 0.25).astype(np.float32)
    vn = np.where(neg, -rng.uniform(0.5, 1, n), 0).astype(np.float32)
    lp = rng.integers(-500, 500, (2, n)).astype(np.int32)
    dev = [torch.from_numpy(x.copy()).cuda() for x in (vp, lp[0], vn, lp[1])]
    wanted = [(np.flatnonzero(pos), vp, lp[0]), (np.flatnonzero(neg), vn, lp[1])]
    cap = max(1, max(w[0].size for w in wanted))
    ws_bytes = lib.seismic_compact_workspace_bytes(n) if with_words else 16 * ((n + 4095) // 4096 + 1)
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    counts = torch.empty(2, dtype=torch.int64, device="cuda")
    out = [torch.full((cap,), -7, dtype=t, device="cuda") for t in (torch.int64, torch.float32, torch.int32) * 2]
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (*dev, *out, counts, ws)]
    _lib.check(lib.seismic_compact_pairs_device(*ptr[:4], n, ctypes.c_float(0.4), cap, *ptr[4:10], ptr[10], ptr[11],
                                                ws_bytes, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert counts.tolist() == [w[0].size for w in wanted]
    for (idx, v, lag), (gi, gv, gl) in zip(wanted, (out[:3], out[3:])):
        np.testing.assert_array_equal(gi.cpu().numpy()[:idx.size], idx)
        np.testing.assert_array_equal(gv.cpu().numpy()[:idx.size], v[idx])
        np.testing.assert_array_equal(gl.cpu().numpy()[:idx.size], lag[idx])
        assert (gi.cpu().numpy()[idx.size:] == -7).all()
