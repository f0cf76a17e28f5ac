"""The division-free histogram bin (csrc/hist_bin.cuh, compiled for the host) against the division, around every bin edge."""
import os
import subprocess

from conftest import ROOT

MAIN = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "hist_bin.cuh"
using namespace seismic;
static long long bad = 0, tried = 0;
static void check(float v, float delta, float inv, int n) {
  ++tried;
  if (hist_bin(v, delta, inv, n) != hist_bin_div(v, delta, n) && bad++ < 5) printf("%.9g at %d bins\n", v, n);
}
static float shift_ulps(float v, int k) {
  int32_t b;
  memcpy(&b, &v, 4);
  b += k;
  if (b < 0) b = 0;
  memcpy(&v, &b, 4);
  return v;
}
int main() {
  const int more[] = {1999, 4096, 4097, 5000, 10007, 20000};
  for (int t = 1; t <= 1200 + 6; ++t) {
    const int n = t <= 1200 ? t : more[t - 1201];
    const float delta = (float)(1.0 / n), inv = 1.0f / delta;
    for (int k = 0; k <= n; ++k) {
      const float a = (float)((double)k * delta), b = (float)((double)k / n);
      for (int u = -8; u <= 8; ++u) {
        check(shift_ulps(a, u), delta, inv, n);
        check(shift_ulps(b, u), delta, inv, n);
      }
    }
    uint32_t x = 12345u + n;
    for (int r = 0; r < 5000; ++r) {
      x = x * 1664525u + 1013904223u;
      check((float)(x >> 8) / 16777216.0f, delta, inv, n);
      check(shift_ulps(0.0f, (int)(x >> 2)), delta, inv, n);  // any exponent, subnormals too
    }
    check(-0.0f, delta, inv, n);
    check(1.0f, delta, inv, n);
    check(1.0000001f, delta, inv, n);
    check(-0.25f, delta, inv, n);
  }
  printf("%lld of %lld differ\n", bad, tried);
  return bad != 0;
}
"""


def test_bins_are_those_of_the_division(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "bins")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "seismic_gb300", "csrc"),
                    str(tmp_path / "main.cpp"), "-o", exe, "-lm"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
