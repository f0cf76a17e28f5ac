"""A tuned slot length is the one that runs: a cached 2, 4 or 8 chunks, the file that the tuner writes, and equal results."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
import torch
from seismic_gb300 import batch, synth, xcorr
for n, c, length, shift, P in ((90, 1, 512, 512, 1024), (60, 3, 500, 512, 1024), (50, 1, 1024, 1024, 2048)):
    ev = torch.from_numpy(synth.family_catalog(n, c, length, n_families=3, seed=n)).cuda()
    for form in ("fp32", "fp16"):
        r = xcorr.xcorr(ev, shift, n_classes_hist=16, form=form)
        for t in (r.vals_pos, r.lags_pos, r.vals_neg, r.lags_neg, r.max_hist, r.min_hist):
            sys.stdout.write("%d " % hash(t.cpu().numpy().tobytes()))
print(batch.tuning(1024, 1)["staged_slot"])
"""


def _run(env):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONHASHSEED": "0", **env})
    assert r.returncode == 0, r.stderr
    *results, slot = r.stdout.split()
    return results, int(slot)


def test_results_do_not_depend_on_the_cached_slots(cuda_ok, tmp_path):
    want, _ = _run({"SEISMIC_TUNE_CACHE": str(tmp_path / "none.txt")})
    for slot in (2, 4, 8):
        f = tmp_path / f"tune{slot}.txt"
        f.write_text("".join(f"P={P} C={c} tile=8 ctas=1 item=16 us=1.0 gpu=x warps=99 ru={min(slot, 4)} slot={slot} rev=2\n"
                             for P in (1024, 2048) for c in (1, 3)))
        got, cached = _run({"SEISMIC_TUNE_CACHE": str(f)})
        assert got == want and cached == slot


def test_the_tuner_writes_the_chunks_that_ran(cuda_ok, tmp_path):
    path = tmp_path / "tune.txt"
    code = (f"from seismic_gb300 import batch; t = batch.autotune(1024, 3, {str(path)!r}); "
            "assert t['staged_slot'] in (2, 4, 8) and t['staged_ru'] == min(t['staged_slot'], 4), t; print(t['staged_slot'])")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SEISMIC_TUNE_CACHE": str(path)})
    assert r.returncode == 0, r.stderr
    assert f"slot={r.stdout.strip()} rev=2" in path.read_text()
