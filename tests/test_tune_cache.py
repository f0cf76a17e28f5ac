"""The autotuner's cache file: what its lines hold is what is reported and used, and shapes timed on a former kernel are not."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

SCRIPT = "import json; from seismic_gb300 import batch; print(json.dumps(batch.tuning(1024, 1)))"


def _tuning(path, lines):
    path.write_text(lines)
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SEISMIC_TUNE_CACHE": str(path)})
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout)


HEAD = "P=1024 C=1 tile=4 ctas=2 item=64 us=100.0 gpu=NVIDIA_GB300"


@pytest.mark.parametrize("tail", ["", " warps=12 ru=2", " warps=99 ru=4", " warps=12 ru=2 slot=2 rev=1"])
def test_shapes_of_a_former_kernel_are_not_used(built_lib, tmp_path, tail):
    t = _tuning(tmp_path / "tune.txt", HEAD + tail + "\n")
    assert (t["staged_warps"], t["staged_ru"], t["staged_slot"]) == (0, 0, 0)
    assert (t["tile"], t["ctas_per_sm"], t["item_groups"]) == (4, 2, 64)


@pytest.mark.parametrize("slot,ru", [(2, 2), (4, 4), (8, 4)])
def test_chunks_are_those_of_the_line(built_lib, tmp_path, slot, ru):
    t = _tuning(tmp_path / "tune.txt", HEAD + f" warps=99 ru={ru} slot={slot} rev=2\n")
    assert (t["staged_warps"], t["staged_ru"], t["staged_slot"]) == (99, ru, slot)
