// Histogram bin of a coefficient: Correlation_in_OMP/correlation_c.cpp:116-117,
// :128-129 (the last bin for v >= 1, else int(v / delta), delta = float(1.0 / n)).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SEISMIC_HIST_FN __host__ __device__ __forceinline__
#else  // host tests compile this header alone
#define SEISMIC_HIST_FN inline
#endif

namespace seismic {

// A negative or NaN coefficient counts in bin 0.
SEISMIC_HIST_FN int hist_bin_clamp(int b, int n_hist) { return b > n_hist - 1 ? n_hist - 1 : (b < 0 ? 0 : b); }

// By the division.
SEISMIC_HIST_FN int hist_bin_div(float v, float delta, int n_hist) {
  if (v >= 1.0f) return n_hist - 1;
  return hist_bin_clamp((int)(v / delta), n_hist);
}

// Without it (an IEEE division is 45 instructions, measured): inv is 1 / delta
// rounded, v inv lies within 1.5 ulp of the quotient, and one residual step
// leaves an error far below an ulp before its rounding, the step of
// correctly rounded division (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000", 1990).  That theorem asks for a first
// quotient within 1 ulp, which v inv does not always meet, and the residual of
// a v near 0 can underflow, so the quotient may differ from the division's in
// its last bit; its integer part does not, by enumeration around every bin
// edge for 1 .. 20,000 bins (tests/test_hist_bin_rule.py runs part of it).
SEISMIC_HIST_FN int hist_bin(float v, float delta, float inv, int n_hist) {
  if (v >= 1.0f) return n_hist - 1;
  const float q = v * inv;
  return hist_bin_clamp((int)fmaf(fmaf(-q, delta, v), inv, q), n_hist);
}

}  // namespace seismic
