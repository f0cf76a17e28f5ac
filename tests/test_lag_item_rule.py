"""The lag-GEMM's item-size rule (csrc/lag_items.cuh, host code) at the launches it was measured on."""
import os
import subprocess

import pytest

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "lag_items.cuh"
using namespace seismic;
int main(int argc, char **argv) {
  const long long n = atoll(argv[1]), q = atoll(argv[2]), work = atoll(argv[5]);
  const int jp = atoi(argv[3]), nhl = atoi(argv[4]);
  const int sms = q ? 150 : 152;
  auto tri = [&](int jc) { return lag_triangle_items(n, 128, 0, (n + 127) / 128, jc); };
  auto rect = [&](int jc) { return (n + 127) / 128 * ((q + jc - 1) / jc); };
  printf("%d", q ? lag_item_js(8, jp, nhl, q, work, sms, rect) : lag_item_js(32, jp, nhl, n, work, sms, tri));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "rule")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "seismic_gb300", "csrc"), str(d / "main.cpp"), "-o", exe],
                   check=True)
    return lambda *a: int(subprocess.run([exe, *map(str, a)], check=True, capture_output=True, text=True).stdout)


# n events, queries (0: the triangle), jp, planes, channels, padded samples, padded lags
@pytest.mark.parametrize("n,q,jp,planes,c,samples,lags,want", [
    (7000, 0, 2, 1, 2, 128, 64, 32), (7000, 0, 2, 2, 2, 128, 64, 32), (5000, 0, 2, 1, 2, 128, 64, 32),  # light, nothing to save
    (7000, 0, 2, 1, 1, 320, 64, 32), (7000, 0, 1, 2, 1, 256, 208, 32), (12000, 0, 2, 2, 1, 64, 32, 32),
    (600, 0, 2, 1, 1, 64, 32, 4), (2000, 0, 2, 2, 1, 128, 128, 2), (150, 0, 2, 2, 1, 64, 64, 2),       # light, much to save
    (4001, 0, 1, 2, 1, 1024, 416, 1), (600, 0, 1, 2, 1, 1024, 416, 4), (16384, 0, 1, 1, 1, 1024, 256, 16),  # heavy: unchanged
    (6177, 5, 1, 1, 3, 1024, 512, 2), (50000, 64, 1, 1, 3, 1024, 512, 8)])
def test_item_size(rule, n, q, jp, planes, c, samples, lags, want):
    assert rule(n, q, jp, planes, c * samples * lags) == want


def test_item_sizes_stay_in_range(rule):
    for n in (1, 2, 127, 128, 129, 1000, 100000):
        for q in (0, 1, 3, 64):
            for jp in (1, 2):
                for work in (1, 1 << 16):
                    jc = rule(n, q, jp, 1, work)
                    assert jc % jp == 0 and jp <= jc <= (8 if q else 32), (n, q, jp, jc)
