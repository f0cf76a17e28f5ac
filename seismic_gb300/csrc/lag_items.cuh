// Work items of the lag-GEMM form (host code): how many j's an item takes.
#pragma once

namespace seismic {

// Items of the triangle's blocks [blk_begin, blk_end) of `m` events each, jc
// j's an item: block b's j's are the events b m .. n - 1.
inline long long lag_triangle_items(long long n, int m, long long blk_begin, long long blk_end, int jc) {
  long long items = 0;
  for (long long b = blk_begin; b < blk_end; ++b) items += (n - b * m + jc - 1) / jc;
  return items;
}

// Multiply-adds a pair and product below which a j is light: most of its time
// is then the epilogue and the output lines that items of few j's share.
constexpr long long kLagLightWork = 1 << 16;

// j's per work item: of 32, 16, ... 1 (multiples of jp, at most `most`), the
// largest whose busiest CTA has the least to walk: its items' j's, and a
// twentieth of a j an item with one plane (measured: N=6000, items of 1 for items of
// 32 cost 2.3 % where they save 2.1 % of the j's; with two planes they cost nothing).
// Light j's (`work` multiply-adds, channels x padded samples x padded lags) leave
// the longest item only for one that saves 6 % or more: shorter items there cost up to
// 18 % where they save 1-4 % (N=7000, two channels of 128 samples, +-30 lags, one
// product: items of 32 3.9 ms, of 8 4.6, of 1 4.6; three products 5.0, 5.2, 5.4), while at N=2000 items of
// 4 or 2 save 7-14 % of the time and at N=600 a third.
// The strips and the A ring run on across items.  items(jc) counts the launch's
// items.  5 queries against 6,177 x 3 events (lags +-256) ran as 49 items of 8 on 49 of
// 150 SMs: 198 us, 147 items of 2: 91 us.  Triangle, three products, N=4001: 12.5 ->
// 11.9 ms; N=600 556 -> 256 us.
template <class F>
inline int lag_item_js(int most, int jp, int nhl, long long j_rows, long long work, int sm_count, F items) {
  int best = jp, longest = 0;
  long long best_cost = -1, longest_cost = 0;
  for (int jc = 32; jc >= jp; jc >>= 1) {
    if (jc > most || jc % jp != 0) continue;
    const long long n = items(jc);
    const long long grid = n < sm_count ? n : sm_count;
    if (grid <= 0) return jc;
    const long long cost = (n + grid - 1) / grid * (20 * (jc < j_rows ? jc : j_rows) + (nhl == 1 ? 1 : 0));
    if (longest == 0) {
      longest = jc;
      longest_cost = cost;
    }
    if (best_cost < 0 || cost < best_cost) {
      best = jc;
      best_cost = cost;
    }
  }
  if (longest != 0 && work < kLagLightWork && 100 * best_cost > 94 * longest_cost) best = longest;
  return best;
}

}  // namespace seismic
