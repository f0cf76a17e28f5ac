"""Server creation where a set-up call fails: a stand-in for cudaFuncSetAttribute refuses the top-K kernel's shared memory."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <dlfcn.h>
#include <stdlib.h>
int cudaFuncSetAttribute(const void *func, int attr, int value) {
  if (attr == 8 && value == 65536 && getenv("REFUSE_64K")) return 1; /* cudaErrorInvalidValue */
  void *h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
  int (*real)(const void *, int, int) = h ? (int (*)(const void *, int, int))dlsym(h, "cudaFuncSetAttribute") : 0;
  return real ? real(func, attr, value) : 999;
}
"""

SCRIPT = r"""
import os
from seismic_gb300 import _lib, serving, synth
cat = synth.ricker_catalog(12, 64, seed=3)
os.environ["REFUSE_64K"] = "1"
try:
    serving.Server(cat, shift=16, form="fp32", topk=4)
    raise SystemExit("created without its top-K kernel")
except _lib.SeismicError as e:
    print("refused:", e)
plain = serving.Server(cat, shift=16, form="fp32", topk=0)  # launches no top-K kernel
assert plain.wait(plain.submit(cat[:2])).vals_pos.shape == (2, 12)
plain.close()
del os.environ["REFUSE_64K"]
srv = serving.Server(cat, shift=16, form="fp32", topk=4)
assert srv.wait(srv.submit(cat[:2])).topk_index[:, 0].tolist() == [0, 1]
srv.close()
print("done")
"""


def test_creation_fails_with_its_cuda_error(cuda_ok, tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    so = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(tmp_path / "shim.c"), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "LD_PRELOAD": so})
    assert r.returncode == 0 and "refused:" in r.stdout and "done" in r.stdout, r.stdout + r.stderr
