// Consumers of the packed outputs: on-device compaction of the pairs above a
// threshold (the reference's sparse output), and a standalone histogram of
// stored coefficients.
//
// The reference thresholds inside the pair loop and then stores each packed
// array as a 1 x N(N+1)/2 CSR matrix of its nonzeros
// (Correlation_in_OMP/test_c.py:43-55, scipy csr_matrix + save_npz).  Here the
// pair kernel can run once with threshold 0; seismic_histogram_device bins the
// stored coefficients with the pair kernel's rule (Correlation_in_OMP/
// correlation_c.cpp:116-117, :128-129) so a threshold can be chosen, and
// seismic_compact_pairs_device keeps, in packed order, the pairs whose
// coefficient passes it (vals_pos > thr, vals_neg < -thr) -- the entries the
// reference's CSR matrices hold after a run with that threshold -- so only
// those cross PCIe.
//
// Compaction.  A count pass reads the values once (HBM-bound), keeps one bit a
// pair and side (kept or not) and counts per CTA; the write pass, whose CTAs
// own the same pairs, sums the counts before its own, reads the bits, 1/32 of
// the values' bytes, and touches only the kept pairs.  Output order is the
// packed order.
#include <cstdint>
#include <type_traits>

#include "../../include/seismic_gb300.h"
#include "hist_bin.cuh"
#include "kernels.cuh"

namespace seismic {

int report_status(int status, const char *message);
int report_cuda(cudaError_t e, const char *what);
void note_launches(unsigned n);

constexpr int kCompactThreads = 256;
constexpr int kCompactWarps = kCompactThreads / 32;
constexpr int kCompactWords = 16;                                     // 32-pair words a warp and side
// Kept pairs of a chunk's 1024 (both sides) from which its 32 words are gone
// through one by one, a bit a lane, instead of finding each round's pairs (16 rounds
// of the search cost what 32 words do: 16.8 M pairs, all kept, 262 us by
// search and 201 by words; a fifth kept 102.5 and, from 256 on by words, 106).
constexpr int kCompactDense = 512;
constexpr int kCompactBlock = kCompactWarps * kCompactWords * 32;     // pairs per block
constexpr int kHistThreads = 256;
constexpr int kHistSmemMax = 4096;
constexpr int kHistSmemBytes = 48 * 1024;

// The blocks that this CTA owns, a contiguous run; warp w takes chunk (512
// pairs) w of each, so a CTA reads 16 KB runs (a run of chunks per warp read 134
// M pairs 20 % slower).
struct CompactRange {
  long long b0, b1;
};
__device__ __forceinline__ CompactRange compact_range(long long nb) {
  return CompactRange{(long long)blockIdx.x * nb / gridDim.x, (long long)(blockIdx.x + 1) * nb / gridDim.x};
}

// Word of this lane in chunk q: the kept bits of 32 consecutive pairs, the
// chunk's positive word `lane` for lane < 16, its negative word lane - 16 for
// the others.
__device__ __forceinline__ unsigned compact_word(const float *__restrict__ vp, const float *__restrict__ vn,
                                                 long long n, float thr, long long q, int lane) {
  const long long e0 = q * kCompactWords * 32 + lane;
  float p[kCompactWords], m[kCompactWords];
#pragma unroll
  for (int k = 0; k < kCompactWords; ++k) {  // 32 loads in flight a thread
    const long long e = e0 + 32 * k;
    p[k] = e < n ? __ldcs(vp + e) : 0.f;
    m[k] = e < n ? __ldcs(vn + e) : 0.f;
  }
  unsigned word = 0;
#pragma unroll
  for (int k = 0; k < kCompactWords; ++k) {
    const bool in = e0 + 32 * k < n;
    const unsigned bp = __ballot_sync(0xffffffffu, in && p[k] > thr);
    const unsigned bn = __ballot_sync(0xffffffffu, in && m[k] < -thr);
    if (lane == k) word = bp;
    if (lane == k + kCompactWords) word = bn;
  }
  return word;
}

// The CTA's sum of a number a warp.  (A 64-bit shared atomicAdd a thread is a
// loop that 256 threads run one after another: 8 us of a small call.)
__device__ __forceinline__ long long warps_sum(const long long (&v)[kCompactWarps]) {
  long long t = 0;
#pragma unroll
  for (int w = 0; w < kCompactWarps; ++w) t += v[w];
  return t;
}

// What bounds it: the read of both value arrays (134 M pairs: 168 us, 6.4 TB/s).
// counts: [2][grid] kept pairs per CTA; totals: zeroed by the caller.
__global__ void __launch_bounds__(kCompactThreads) compact_count_kernel(const float *__restrict__ vp,
                                                                          const float *__restrict__ vn,
                                                                          long long n, float thr, long long nb,
                                                                          long long *__restrict__ counts,
                                                                          unsigned *__restrict__ words,
                                                                          unsigned long long *__restrict__ totals) {
  __shared__ long long s_cnt[2][kCompactWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const CompactRange r = compact_range(nb);
  long long mine = 0;
  for (long long b = r.b0; b < r.b1; ++b) {
    const long long q = b * kCompactWarps + warp;
    const unsigned word = compact_word(vp, vn, n, thr, q, lane);
    if (words) words[q * 32 + lane] = word;
    mine += __popc(word);
  }
  for (int o = kCompactWords / 2; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if (lane % kCompactWords == 0) s_cnt[lane / kCompactWords][warp] = mine;
  __syncthreads();
  if (threadIdx.x < 2) {
    const long long all = warps_sum(s_cnt[threadIdx.x]);
    counts[(long long)threadIdx.x * gridDim.x + blockIdx.x] = all;
    if (all) atomicAdd(&totals[threadIdx.x], (unsigned long long)all);
  }
}

// The kept pairs of each chunk, one a lane: lane s takes the chunk's s-th kept
// pair (a search over the words' running counts, then the bit of its rank), so
// up to 32 gathers are in flight a warp and the stores are contiguous however
// many are kept; a chunk with kCompactDense kept pairs or more goes word by word
// instead.  134 M pairs, 2 % kept: 205 us (count and write 317) against 1514 with two
// barriers per 256 pairs and 428 with a word at a time.  Small calls: a 64-bit shared atomicAdd a
// thread for the counts of the CTAs before this one cost more than the gathers
// (1 M pairs, count and write, 2 % kept 38.5 us, all kept 61; now 18 and 27).  WORDS: the stored
// words are read, by 8 CTAs an SM (the whole grid resident; two rounds at a time and
// 5 CTAs: 339 us).  Without them (a workspace that has no room) the values are
// read again, 32 loads in flight a thread, which takes the registers of 5 CTAs.
template <bool WORDS>
__global__ void __launch_bounds__(kCompactThreads, WORDS ? 8 : 5) compact_write_kernel(
    const float *__restrict__ vp, const int *__restrict__ lp, const float *__restrict__ vn,
    const int *__restrict__ ln, long long n, float thr, long long nb, const long long *__restrict__ counts,
    const unsigned *__restrict__ words, long long capacity, long long *__restrict__ idx_p,
    float *__restrict__ val_p, int *__restrict__ lag_p, long long *__restrict__ idx_n, float *__restrict__ val_n,
    int *__restrict__ lag_n) {
  __shared__ long long s_before[2][kCompactWarps];  // kept pairs of the CTAs before this one, by warp
  __shared__ int s_warp[2][2][kCompactWarps];       // [block parity][side]: of each warp's chunk
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long before[2] = {0, 0};
  for (int c = threadIdx.x; c < (int)blockIdx.x; c += kCompactThreads) {
    before[0] += counts[c];
    before[1] += counts[(long long)gridDim.x + c];
  }
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    for (int o = 16; o > 0; o >>= 1) before[sd] += __shfl_xor_sync(0xffffffffu, before[sd], o);
    if (lane == 0) s_before[sd][warp] = before[sd];
  }
  __syncthreads();
  long long off_p = warps_sum(s_before[0]), off_n = warps_sum(s_before[1]);
  const CompactRange r = compact_range(nb);
  for (long long b = r.b0; b < r.b1; ++b) {
    const long long q = b * kCompactWarps + warp;
    const unsigned word = WORDS ? __ldg(words + q * 32 + lane) : compact_word(vp, vn, n, thr, q, lane);
    const int c = __popc(word);
    int incl = c;  // running count over the 16 positive words, then the 16 negative ones
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    const int pos = __shfl_sync(0xffffffffu, incl, kCompactWords - 1), all = __shfl_sync(0xffffffffu, incl, 31);
    int(&cnt)[2][kCompactWarps] = s_warp[b & 1];  // two sets: the next block's is written while this one is read
    if (lane == 0) {
      cnt[0][warp] = pos;
      cnt[1][warp] = all - pos;
    }
    __syncthreads();
    long long at_p = off_p, at_n = off_n;  // this chunk's first positive and negative pair
    for (int w = 0; w < kCompactWarps; ++w) {
      off_p += cnt[0][w];
      off_n += cnt[1][w];
      if (w < warp) {
        at_p += cnt[0][w];
        at_n += cnt[1][w];
      }
    }
    // rounds of up to 32 kept pairs, U at a time: their gathers are issued before the first store
    auto rounds = [&](auto by_word, int n_rounds) {
      constexpr int U = WORDS ? 1 : 2;
      for (int r0 = 0; r0 < n_rounds; r0 += U) {
        int at[U], rank[U];  // the pair within the chunk (word and bit; -1: none), and its rank among the kept
        float val[U];
        int lag[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          at[u] = -1;
          if (U > 1 && r0 + u >= n_rounds) continue;  // uniform
          int k, bit, s;
          bool kept;
          if constexpr (by_word.value) {
            k = r0 + u;
            bit = lane;
            const unsigned bits = __shfl_sync(0xffffffffu, word, k);
            s = __shfl_sync(0xffffffffu, incl, k) - __popc(bits) + __popc(bits & ((1u << lane) - 1u));
            kept = (bits >> lane) & 1u;
          } else {
            s = 32 * (r0 + u) + lane;
            kept = s < all;
            k = 0;  // the word of the s-th kept pair: words whose running count is <= s
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) {
              const int x = __shfl_sync(0xffffffffu, incl, k + w - 1);
              if (x <= s) k += w;
            }
            k = k < 31 ? k : 31;
            const unsigned bits = __shfl_sync(0xffffffffu, word, k);
            int left = s - (__shfl_sync(0xffffffffu, incl, k) - __popc(bits));
            bit = 0;  // the set bit of that rank
#pragma unroll
            for (int w = 16; w > 0; w >>= 1) {
              const int x = __popc((bits >> bit) & ((1u << w) - 1u));
              if (left >= x) {
                left -= x;
                bit += w;
              }
            }
          }
          const bool neg = s >= pos;
          const int c = (k & (kCompactWords - 1)) * 32 + bit;
          const long long e = q * (kCompactWords * 32) + c, o = neg ? at_n + (s - pos) : at_p + s;
          // (e and o lie in range whenever the counts and words are those of these arrays)
          if (kept && e < n && o >= 0 && o < capacity) {
            at[u] = c;
            rank[u] = s;
            val[u] = __ldg((neg ? vn : vp) + e);
            lag[u] = __ldg((neg ? ln : lp) + e);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (at[u] >= 0) {
            const bool neg = rank[u] >= pos;
            const long long o = neg ? at_n + (rank[u] - pos) : at_p + rank[u];
            (neg ? idx_n : idx_p)[o] = q * (kCompactWords * 32) + at[u];
            (neg ? val_n : val_p)[o] = val[u];
            (neg ? lag_n : lag_p)[o] = lag[u];
          }
        }
      }
    };
    if (all == 0) continue;  // uniform over the warp
    if (all >= kCompactDense) rounds(std::true_type{}, 32);
    else rounds(std::false_type{}, (all + 31) / 32);
  }
}

// Histograms in shared memory, `rep` copies of each counter (a power of two up
// to 32) used by lane % rep: the coefficients of a catalog fall into a few
// bins, and a warp's 32 additions to the same few words ran one after another.
// Four loads an array in flight a thread.  134 M pairs, 20 bins: 178 us against
// 469 with one copy and a division a value.  Adding the copies up with all lanes
// at the same copy was a bank conflict of up to `rep` ways: 1 M pairs, 100 bins, 32 us,
// now 13 (16 with one copy).
__global__ void __launch_bounds__(kHistThreads) histogram_kernel(const float *__restrict__ vp,
                                                                 const float *__restrict__ vn, long long n,
                                                                 int n_hist, float delta, float inv, int rep,
                                                                 int *hmax, int *hmin) {
  extern __shared__ __align__(8) int s_hist[];  // [2][n_hist][rep]; rep == 0: counted in global memory
  for (int h = threadIdx.x; h < n_hist * rep; h += blockDim.x) reinterpret_cast<int2 *>(s_hist)[h] = make_int2(0, 0);
  __syncthreads();
  const int mine = rep ? (int)threadIdx.x & (rep - 1) : 0;
  auto count = [&](float p, float m) {
    const int hp = hist_bin(p, delta, inv, n_hist);
    const int hn = hist_bin(-m, delta, inv, n_hist);
    if (rep) {
      atomicAdd(&s_hist[hp * rep + mine], 1);
      atomicAdd(&s_hist[(n_hist + hn) * rep + mine], 1);
    } else {
      atomicAdd(&hmax[hp], 1);
      atomicAdd(&hmin[hn], 1);
    }
  };
  constexpr int U = 4;
  const long long step = (long long)gridDim.x * kHistThreads * U;
  long long e = (long long)blockIdx.x * kHistThreads * U + threadIdx.x;
  for (; e + (U - 1) * kHistThreads < n; e += step) {
    float p[U], m[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      p[k] = __ldcs(vp + e + k * kHistThreads);
      m[k] = __ldcs(vn + e + k * kHistThreads);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) count(p[k], m[k]);
  }
  for (; e < n; e += kHistThreads) count(__ldcs(vp + e), __ldcs(vn + e));  // the last, partial batch
  __syncthreads();
  if (rep) {
    // each lane starts at another copy: bins lie `rep` words apart, so the same copy
    // of 32 bins would be 32 words of one bank
    const int turn = (int)(threadIdx.x & 31) * rep / 32;
    for (int h = threadIdx.x; h < n_hist; h += blockDim.x) {
      int tp = 0, tn = 0;
#pragma unroll 4
      for (int r = 0; r < rep; ++r) {
        const int c = (r + turn) & (rep - 1);
        tp += s_hist[h * rep + c];
        tn += s_hist[(n_hist + h) * rep + c];
      }
      if (tp) atomicAdd(&hmax[h], tp);
      if (tn) atomicAdd(&hmin[h], tn);
    }
  }
}

// Workspace: the counts per CTA (at most nb CTAs, 2 nb words of 8 bytes), then
// (where there is room) the words.
long long compact_blocks(long long n) { return (n + kCompactBlock - 1) / kCompactBlock; }
size_t compact_count_bytes(long long nb) { return (size_t)(2 * nb + 2) * sizeof(long long); }
size_t compact_bytes(long long nb) {
  return compact_count_bytes(nb) + (size_t)nb * kCompactWarps * 32 * sizeof(unsigned);
}

}  // namespace seismic

using namespace seismic;

extern "C" {

size_t seismic_compact_workspace_bytes(long long n_pairs) {
  if (n_pairs < 0) return 0;
  return compact_bytes(compact_blocks(n_pairs));
}

// Both compaction calls: `count` runs the count pass, `capacity` >
// 0 the write pass.
static int compact_run(const float *d_vals_pos, const int *d_lags_pos, const float *d_vals_neg,
                       const int *d_lags_neg, long long n_pairs, float threshold, long long capacity,
                       long long *d_index_pos, float *d_value_pos, int *d_lag_pos, long long *d_index_neg,
                       float *d_value_neg, int *d_lag_neg, long long *d_counts, void *workspace,
                       size_t workspace_bytes, void *stream, bool count) {
  report_status(SEISMIC_OK, "");
  if (n_pairs < 0 || capacity < 0 || !(threshold >= 0.f))
    return report_status(SEISMIC_ERR_INVALID_ARGUMENT, "n_pairs, capacity and threshold must be >= 0");
  if (!d_vals_pos || !d_lags_pos || !d_vals_neg || !d_lags_neg || (count && !d_counts) || !workspace)
    return report_status(SEISMIC_ERR_INVALID_ARGUMENT, "null buffer");
  if (capacity > 0 && (!d_index_pos || !d_value_pos || !d_lag_pos || !d_index_neg || !d_value_neg || !d_lag_neg))
    return report_status(SEISMIC_ERR_INVALID_ARGUMENT, "null output buffer with capacity > 0");
  const long long nb = compact_blocks(n_pairs);
  // a workspace with room for the block counts alone is taken too; the write
  // pass then reads the values again
  if (workspace_bytes < compact_count_bytes(nb))
    return report_status(SEISMIC_ERR_WORKSPACE_TOO_SMALL, "compaction workspace too small");
  int sm = 0;
  const float2 *tw;
  int *ef;
  int s = device_context(&sm, &tw, &ef);
  if (s) return s;
  cudaStream_t st = (cudaStream_t)stream;
  long long *counts = static_cast<long long *>(workspace);
  unsigned *words = workspace_bytes < compact_bytes(nb) ? nullptr
                                                        : reinterpret_cast<unsigned *>(counts + 2 * nb + 2);
  cudaError_t e = cudaSuccess;
  if (nb == 0) {
    if (count) e = cudaMemsetAsync(d_counts, 0, 2 * sizeof(long long), st);
    return e == cudaSuccess ? SEISMIC_OK : report_cuda(e, "compaction count clear");
  }
  // the same grid in both passes: a CTA of the write pass owns the pairs that
  // its count covers
  const int grid = (int)(nb < (long long)sm * 8 ? nb : (long long)sm * 8);
  if (count) {
    e = cudaMemsetAsync(d_counts, 0, 2 * sizeof(long long), st);
    if (e != cudaSuccess) return report_cuda(e, "compaction count clear");
    compact_count_kernel<<<grid, kCompactThreads, 0, st>>>(d_vals_pos, d_vals_neg, n_pairs, threshold, nb, counts,
                                                           words, reinterpret_cast<unsigned long long *>(d_counts));
    e = cudaGetLastError();
    note_launches(1);
  }
  if (e == cudaSuccess && capacity > 0) {
    const auto write = words ? compact_write_kernel<true> : compact_write_kernel<false>;
    write<<<grid, kCompactThreads, 0, st>>>(d_vals_pos, d_lags_pos, d_vals_neg, d_lags_neg, n_pairs, threshold, nb,
                                            counts, words, capacity, d_index_pos, d_value_pos, d_lag_pos,
                                            d_index_neg, d_value_neg, d_lag_neg);
    e = cudaGetLastError();
    note_launches(1);
  }
  return e == cudaSuccess ? SEISMIC_OK : report_cuda(e, "compaction launch");
}

int seismic_compact_pairs_device(const float *d_vals_pos, const int *d_lags_pos, const float *d_vals_neg,
                                 const int *d_lags_neg, long long n_pairs, float threshold, long long capacity,
                                 long long *d_index_pos, float *d_value_pos, int *d_lag_pos,
                                 long long *d_index_neg, float *d_value_neg, int *d_lag_neg,
                                 long long *d_counts, void *workspace, size_t workspace_bytes, void *stream) {
  return compact_run(d_vals_pos, d_lags_pos, d_vals_neg, d_lags_neg, n_pairs, threshold, capacity, d_index_pos,
                     d_value_pos, d_lag_pos, d_index_neg, d_value_neg, d_lag_neg, d_counts, workspace,
                     workspace_bytes, stream, true);
}

int seismic_compact_write_device(const float *d_vals_pos, const int *d_lags_pos, const float *d_vals_neg,
                                 const int *d_lags_neg, long long n_pairs, float threshold, long long capacity,
                                 long long *d_index_pos, float *d_value_pos, int *d_lag_pos,
                                 long long *d_index_neg, float *d_value_neg, int *d_lag_neg,
                                 const void *workspace, size_t workspace_bytes, void *stream) {
  return compact_run(d_vals_pos, d_lags_pos, d_vals_neg, d_lags_neg, n_pairs, threshold, capacity, d_index_pos,
                     d_value_pos, d_lag_pos, d_index_neg, d_value_neg, d_lag_neg, nullptr,
                     const_cast<void *>(workspace), workspace_bytes, stream, false);
}

int seismic_histogram_device(const float *d_vals_pos, const float *d_vals_neg, long long n_pairs,
                             int n_classes_hist, int *d_max_hist, int *d_min_hist, void *stream) {
  report_status(SEISMIC_OK, "");
  if (n_pairs < 0 || n_classes_hist < 1)
    return report_status(SEISMIC_ERR_INVALID_ARGUMENT, "n_pairs must be >= 0 and n_classes_hist >= 1");
  if (!d_vals_pos || !d_vals_neg || !d_max_hist || !d_min_hist)
    return report_status(SEISMIC_ERR_INVALID_ARGUMENT, "null buffer");
  if (n_pairs == 0) return SEISMIC_OK;
  int sm = 0;
  const float2 *tw;
  int *ef;
  int s = device_context(&sm, &tw, &ef);
  if (s) return s;
  const long long want = (n_pairs + 4 * kHistThreads - 1) / (4 * kHistThreads);
  const int grid = (int)(want < (long long)sm * 8 ? want : (long long)sm * 8);
  // copies of the counters: as many as fit the shared memory that every launch
  // may use without an attribute; none (global counters) past kHistSmemMax bins
  int rep = n_classes_hist <= kHistSmemMax ? 32 : 0;
  while (rep > 1 && (size_t)2 * n_classes_hist * rep * sizeof(int) > (size_t)kHistSmemBytes) rep >>= 1;
  const float delta = (float)(1.0 / n_classes_hist);
  histogram_kernel<<<grid, kHistThreads, (size_t)2 * n_classes_hist * rep * sizeof(int), (cudaStream_t)stream>>>(
      d_vals_pos, d_vals_neg, n_pairs, n_classes_hist, delta, 1.0f / delta, rep, d_max_hist, d_min_hist);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return report_cuda(e, "histogram launch");
  note_launches(1);
  return SEISMIC_OK;
}

}  // extern "C"
