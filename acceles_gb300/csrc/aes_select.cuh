// aes_select.cuh -- the stages after the candidate pass of the two-stage Top-K SpMV engine, and
// the query quantiser before it (reference: zhaijiaqi/AccelES):
//   k_quantize        quantify_vector (quantify_util.py:31-49) / quantize_vec
//                     (quantize_utils.hpp:8-18): float64 results in integer arithmetic, one CTA per query
//   k_threshold       per (query, partition) lower bound of the Top-CK boundary from a sample
//   k_select          exact Top-CK per partition, (key desc, row desc)
//                     (split_approximate, quantify_util.py:173-196; sort_tuples order)
//   k_final           FP32 rescoring of the candidates (quantify_util.py:354-356 in FP32;
//                     gold_algorithms.hpp:211-239 summation order) and the final Top-K
//   k_exact_sample, k_exact_all, k_exact_multi   the FP32-only Top-K of every row
#pragma once

#include <algorithm>

#include "aes_kernels.cuh"

namespace aes {
namespace dev {

// ---------------------------------------------------------------------------------------------
// query quantiser: one CTA per query.  The integer query is bit-identical to quantify_vector
// (quantify_util.py:31-49) applied to the float64 upcast of the FP32 query: numpy's binary64
// division and multiplication (round to nearest even) and round-half-to-even are reproduced in
// integer arithmetic (aes_qexact.hpp), so no FP64 runs on the GPU.
// quant: 0 symmetric, 1/2 unsigned (per query); qq: 0 numpy, 1 quantize_vec truncation.
// ---------------------------------------------------------------------------------------------
// threads per query: the rounding is a long chain of 64-bit divisions, so a few queries spread their
// columns wide (1024 columns: 7.6 us with 256 threads, 5.5 with 1024)
__host__ inline unsigned quantize_threads(uint32_t nq) { return nq <= 64 ? 1024u : 256u; }
__global__ void __launch_bounds__(1024) k_quantize(const float* __restrict__ q32, uint32_t cols, uint32_t ld32, int bits,
                           int quant, int qq, int8_t* __restrict__ q8, uint32_t ld8,
                           uint32_t* __restrict__ status, float* __restrict__ copy) {
  grid_wait();
  grid_next();
  __shared__ float red[32];
  __shared__ int negs;
  const float* x = q32 + (size_t)blockIdx.x * ld32;
  int8_t* o = q8 + (size_t)blockIdx.x * ld8;
  if (threadIdx.x == 0) status[blockIdx.x] = 0;
  if (copy) {  // the queries are in pinned host memory: the later stages read them from here
    float* d = copy + (size_t)blockIdx.x * ld32;
    for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) d[j] = x[j];
    x = d;
    __syncthreads();
  }
  if (qq == 1) {  // quantize_utils.hpp:8-18 (ap_fixed<32,B,AP_TRN_ZERO>, to_int, ap_int<B>)
    const int F = 32 - bits;
    for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) {
      const int32_t X32 = qx::trunc_scaled30(x[j]);  // x * 2^(B-2+F), truncated, 32-bit wrap
      int32_t n = X32 / (int32_t)(1u << F);
      int32_t mask = (1 << bits) - 1, half = 1 << (bits - 1);
      o[j] = (int8_t)(((n & mask) ^ half) - half);
    }
    return;
  }
  float m = 0.0f;
  int neg = 0;
  for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) {
    float v = x[j];
    neg |= (v < 0.0f);
    m = fmaxf(m, quant == 0 ? fabsf(v) : v);
  }
  if (threadIdx.x == 0) negs = 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, d));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  if (neg) atomicOr(&negs, 1);
  __syncthreads();
  if (threadIdx.x < 32) {
    float r = threadIdx.x < (blockDim.x + 31) / 32 ? red[threadIdx.x] : 0.0f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) r = fmaxf(r, __shfl_xor_sync(0xFFFFFFFFu, r, d));
    if (threadIdx.x == 0) red[0] = r;
  }
  __syncthreads();
  const float mm = red[0];  // max |x| (or max x)
  if (quant != 0 && negs) {
    if (threadIdx.x == 0) status[blockIdx.x] = ST_QUERY;
    for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) o[j] = 0;
    return;
  }
  const int32_t M = quant == 0 ? ((1 << bits) - 1) / 2 : (1 << bits) - 1;
  const int32_t lo = quant == 0 ? -M - 1 : 0;
  for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) {
    int32_t q = 0;
    if (mm != 0.0f) {
      q = qx::round_scaled(x[j], mm, M);  // the float64 arithmetic of numpy, in integers
      q = q < lo ? lo : (q > M ? M : q);
    }
    o[j] = (int8_t)(uint8_t)(uint32_t)q;
  }
}

// ---------------------------------------------------------------------------------------------
// block helpers
// ---------------------------------------------------------------------------------------------
constexpr int kHistBins = 2048;
constexpr int kThrILP = 12;  // keys in flight per thread in the threshold passes
constexpr int kThreadsThr = 512;  // at most 64 registers: two CTAs per SM, a 256-query batch in one wave

// The bin holding the need-th largest item of a kHistBins histogram (1 <= need <= its total):
// {bin, items above it, items in it}.  Every thread of a THREADS-wide block calls it; sh holds
// THREADS / 32 + 3 words.  Each thread sums its share of the bins, a warp scan and the warps'
// totals give the items above it: two barriers, where one warp walking 64 bins per lane took 2 us.
struct TopBin {
  uint32_t bin, above, in;
};
template <int THREADS>
__device__ __forceinline__ TopBin block_top_bin(const uint32_t* hist, uint32_t need, uint32_t* sh) {
  constexpr int PER = kHistBins / THREADS, NW = THREADS / 32;
  static_assert(PER == 2 || PER == 4 || PER == 8, "bins per thread");
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t h[PER], own = 0;
#pragma unroll
  for (int i = 0; i < PER; i++) {
    h[i] = hist[threadIdx.x * PER + i];
    own += h[i];
  }
  uint32_t incl = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t u = __shfl_down_sync(0xFFFFFFFFu, incl, d);
    if (lane + d < 32) incl += u;
  }
  if (lane == 0) sh[warp] = incl;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NW; w++) incl += w > (int)warp ? sh[w] : 0u;
  uint32_t acc = incl - own;
  if (acc < need && incl >= need) {
    bool found = false;
#pragma unroll
    for (int i = PER - 1; i >= 0; i--) {
      if (!found && acc + h[i] >= need) {
        sh[NW] = threadIdx.x * PER + i;
        sh[NW + 1] = acc;
        sh[NW + 2] = h[i];
        found = true;
      }
      acc += h[i];
    }
  }
  __syncthreads();
  const TopBin r{sh[NW], sh[NW + 1], sh[NW + 2]};
  return r;
}

// The r-th largest (1 <= r <= total) of the keys a warp holds, N per lane (lanes without a key
// hold 0, which is below every real one or equal to it): the largest t with at least r keys >= t,
// found bit by bit below the bits that the smallest and the largest key share.
template <int N>
__device__ __forceinline__ uint32_t warp_rth_key(const uint32_t (&k)[N], uint32_t mn, uint32_t mx,
                                                 uint32_t r) {
  const uint32_t diff = mn ^ mx;
  if (diff == 0) return mn;
  int bit = 31 - __clz(diff);
  uint32_t t = bit == 31 ? 0u : mx & ~((2u << bit) - 1u);
  for (; bit >= 0; bit--) {
    const uint32_t c = t | (1u << bit);
    uint32_t n = 0;
#pragma unroll
    for (int i = 0; i < N; i++) n += k[i] >= c ? 1u : 0u;
    if (__reduce_add_sync(0xFFFFFFFFu, n) >= r) t = c;
  }
  return t;
}

// ---------------------------------------------------------------------------------------------
// k_threshold: per (query, partition), the r-th largest sample key (or a lower bound of it exact
// within 2^shift2), so that every row at or above the partition's Top-CK boundary has a key
// >= L with overwhelming probability; a miss is detected later (ST_MISS) and repaired.
// Also resets the partition's survivor counter.
//
// Latency-bound: a few thousand keys from L2 per partition, and a select.  Two forms:
// k_threshold_warp, one warp per (query, partition), where no partition has more than
// kThrWarpKeys samples: the keys stay in registers (100 queries x 32 partitions of 195 samples:
// 43 -> 6.7 us); k_threshold, one CTA each, for the rest.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kThrWarpKeys = 1024;  // 32 per lane (16 for half as many)
constexpr int kThrWarps = 4;             // (query, partition) pairs per CTA
constexpr uint32_t kThrRankMax = 128;    // ranks up to which the CTA form selects by group maxima
constexpr uint32_t kThrListMax = 1024;

template <int N>
__global__ void __launch_bounds__(kThrWarps * 32) k_threshold_warp(
    const uint32_t* keys_all, uint32_t ld_keys, const uint32_t* __restrict__ part_begin,
    uint32_t split, uint32_t pairs, const uint32_t* __restrict__ r_part, uint32_t* __restrict__ thr,
    uint32_t* __restrict__ cnt) {
  grid_wait();
  grid_next();
  const uint32_t i = blockIdx.x * kThrWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  if (i >= pairs) return;
  const uint32_t p = i % split, q = i / split;
  const uint32_t a = __ldg(part_begin + p), n = __ldg(part_begin + p + 1) - a, r = __ldg(r_part + p);
  const uint32_t* kb = keys_all + (size_t)q * ld_keys + a;
  uint32_t k[N], mn = 0xFFFFFFFFu, mx = 0;
#pragma unroll
  for (int u = 0; u < N; u++) {
    const uint32_t j = u * 32 + lane;
    k[u] = j < n ? kb[j] : 0u;
    if (j < n) {
      mn = min(mn, k[u]);
      mx = max(mx, k[u]);
    }
  }
  mn = __reduce_min_sync(0xFFFFFFFFu, mn);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  // too few samples: keep every row of the partition
  const uint32_t t = (n < r || r == 0) ? 0u : warp_rth_key<N>(k, mn, mx, r);
  if (lane == 0) {
    thr[i] = t;
    cnt[i] = 0;
  }
}

// Sample keys of query q: keys_all[q * ld_keys + i].
//
// Ranks up to kThrRankMax: every thread's largest key is found in one pass; the r-th largest of
// those maxima (of groups of two or four threads where r is small) is a bound that r keys reach and
// few others do, so the few threads at or above it gather their keys of at least that bound, and
// the r-th largest of the gathered keys is the answer.  One read of the keys, where two
// histograms took three: 27 -> 12.8 us for 39k keys, r = 24.  Larger ranks: two histograms.
__global__ void __launch_bounds__(kThreadsThr, 2) k_threshold(const uint32_t* keys_all, uint32_t ld_keys,
                            const uint32_t* __restrict__ part_begin, uint32_t split,
                            const uint32_t* __restrict__ r_part, uint32_t* __restrict__ thr,
                            uint32_t* __restrict__ cnt) {
  grid_wait();
  grid_next();
  __shared__ __align__(16) uint32_t hist[kHistBins];
  __shared__ uint32_t smin[kThreadsThr / 32], smax[kThreadsThr / 32], sh[kThreadsThr / 32 + 3];
  __shared__ uint32_t s_bound, s_n;
  const uint32_t p = blockIdx.x, q = blockIdx.y;
  const uint32_t* kk = keys_all + (size_t)q * ld_keys;
  const uint32_t a = part_begin[p], b = part_begin[p + 1];
  const uint32_t n = b - a;
  const uint32_t r = r_part[p];
  uint32_t* T = thr + (size_t)q * split + p;
  if (threadIdx.x == 0) cnt[(size_t)q * split + p] = 0;
  if (n < r || r == 0) {
    if (threadIdx.x == 0) *T = 0;  // too few samples: keep every row of the partition
    return;
  }
  // every pass reads several keys per thread before using them: the loops are bound by global
  // load latency otherwise
  uint32_t mn = 0xFFFFFFFFu, mx = 0;
  for (uint32_t i0 = a; i0 < b; i0 += kThreadsThr * kThrILP) {
    uint32_t v[kThrILP];
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      v[u] = i < b ? kk[i] : 0u;
    }
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      if (i < b) {
        mn = min(mn, v[u]);
        mx = max(mx, v[u]);
      }
    }
  }
  if (r <= kThrRankMax && n >= (uint32_t)kThreadsThr) {
    const uint32_t own = mx;
    uint32_t* gm = hist;  // group maxima
    uint32_t per = 1;     // threads per maximum: 128 groups are enough for r <= 32, 256 for 64
    uint32_t g = mx;
    if (r <= 64u) {
      per = 2;
      g = max(g, __shfl_xor_sync(0xFFFFFFFFu, g, 1));
    }
    if (r <= 32u) {
      per = 4;
      g = max(g, __shfl_xor_sync(0xFFFFFFFFu, g, 2));
    }
    const uint32_t ng = kThreadsThr / per, mine = threadIdx.x / per;
    if (threadIdx.x % per == 0) gm[mine] = g;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    uint32_t gt = 0, ge = 0;
    for (uint32_t j = threadIdx.x % per; j < ng; j += per) {
      gt += gm[j] > g ? 1u : 0u;
      ge += gm[j] >= g ? 1u : 0u;
    }
    for (uint32_t d = per >> 1; d > 0; d >>= 1) {
      gt += __shfl_xor_sync(0xFFFFFFFFu, gt, d);
      ge += __shfl_xor_sync(0xFFFFFFFFu, ge, d);
    }
    if (gt < r && ge >= r) s_bound = g;  // (the same value from every thread that gets here)
    __syncthreads();
    const uint32_t bound = s_bound;
    uint32_t* list = hist + kThreadsThr;  // kThrListMax keys
    if (own >= bound) {
      for (uint32_t i0 = a; i0 < b; i0 += kThreadsThr * kThrILP) {
        uint32_t v[kThrILP];
#pragma unroll
        for (int u = 0; u < kThrILP; u++) {
          const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
          v[u] = i < b ? kk[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < kThrILP; u++) {
          const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
          if (i < b && v[u] >= bound) {
            const uint32_t o = atomicAdd(&s_n, 1u);
            if (o < kThrListMax) list[o] = v[u];
          }
        }
      }
    }
    __syncthreads();
    const uint32_t m = s_n;  // >= r
    if (m <= kThrListMax) {
      for (uint32_t i = threadIdx.x; i < m; i += kThreadsThr) {
        const uint32_t v = list[i];
        uint32_t lgt = 0, lge = 0;
        for (uint32_t j = 0; j < m; j++) {
          lgt += list[j] > v ? 1u : 0u;
          lge += list[j] >= v ? 1u : 0u;
        }
        if (lgt < r && lge >= r) *T = v;
      }
      return;
    }
    __syncthreads();  // many equal keys: the histograms below
  }
  mn = __reduce_min_sync(0xFFFFFFFFu, mn);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  if ((threadIdx.x & 31) == 0) { smin[threadIdx.x >> 5] = mn; smax[threadIdx.x >> 5] = mx; }
  for (int i = threadIdx.x; i < kHistBins; i += kThreadsThr) hist[i] = 0;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreadsThr / 32; w++) {
    mn = min(mn, smin[w]);
    mx = max(mx, smax[w]);
  }
  const uint32_t span = mx - mn;
  if (span == 0) {
    if (threadIdx.x == 0) *T = mn;
    return;
  }
  const int bl = 32 - __clz(span);           // bits of span
  const int sh1 = bl > 11 ? bl - 11 : 0;
  for (uint32_t i0 = a; i0 < b; i0 += kThreadsThr * kThrILP) {
    uint32_t v[kThrILP];
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      v[u] = i < b ? kk[i] : 0u;
    }
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      if (i < b) atomicAdd(&hist[(v[u] - mn) >> sh1], 1u);
    }
  }
  __syncthreads();
  const TopBin t1 = block_top_bin<kThreadsThr>(hist, r, sh);
  if (sh1 == 0) {
    if (threadIdx.x == 0) *T = mn + t1.bin;
    return;
  }
  const int sh2 = sh1 > 11 ? sh1 - 11 : 0;
  for (int i = threadIdx.x; i < kHistBins; i += kThreadsThr) hist[i] = 0;
  __syncthreads();
  for (uint32_t i0 = a; i0 < b; i0 += kThreadsThr * kThrILP) {
    uint32_t v[kThrILP];
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      v[u] = i < b ? kk[i] : 0u;
    }
#pragma unroll
    for (int u = 0; u < kThrILP; u++) {
      const uint32_t i = i0 + u * kThreadsThr + threadIdx.x;
      if ((i < b) && (((v[u] - mn) >> sh1) == t1.bin))
        atomicAdd(&hist[((v[u] - mn) >> sh2) & ((1u << (sh1 - sh2)) - 1u)], 1u);
    }
  }
  __syncthreads();
  const TopBin t2 = block_top_bin<kThreadsThr>(hist, r - t1.above, sh);
  if (threadIdx.x == 0) *T = mn + (t1.bin << sh1) + (t2.bin << sh2);
}

// ---------------------------------------------------------------------------------------------
// Block-wide exact select: the `need` largest 64-bit composites (key << 32 | row) of n items.
// Items come from an accessor; returns through smem the threshold composite tau such that
// exactly `need` items are >= tau (composites are unique because rows are).
// ---------------------------------------------------------------------------------------------
template <class Get>
__device__ uint64_t block_select_tau(Get get, uint32_t n, uint32_t need, uint32_t* hist256,
                                     uint64_t* sh64) {
  // min / max composite
  uint64_t mn = ~0ull, mx = 0;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    uint64_t c = get(i);
    mn = c < mn ? c : mn;
    mx = c > mx ? c : mx;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    uint64_t a = __shfl_xor_sync(0xFFFFFFFFu, mn, d), b = __shfl_xor_sync(0xFFFFFFFFu, mx, d);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) { sh64[threadIdx.x >> 5] = mn; sh64[32 + (threadIdx.x >> 5)] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t nw = (blockDim.x + 31) / 32;
    uint64_t a = ~0ull, b = 0;
    for (uint32_t w = 0; w < nw; w++) {
      a = sh64[w] < a ? sh64[w] : a;
      b = sh64[32 + w] > b ? sh64[32 + w] : b;
    }
    sh64[64] = a;
    sh64[65] = b;
  }
  __syncthreads();
  mn = sh64[64];
  mx = sh64[65];
  if (need >= n) return mn;
  if (mn == mx) return mn;
  int hi = 63 - __clzll((long long)(mn ^ mx));
  uint64_t prefix = mx & ~((hi == 63) ? ~0ull : ((2ull << hi) - 1ull));
  uint64_t fixed = ~((hi == 63) ? ~0ull : ((2ull << hi) - 1ull));
  uint32_t need_rem = need;
  while (true) {
    const int lo = hi >= 7 ? hi - 7 : 0;
    const int width = hi - lo + 1;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) hist256[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      uint64_t c = get(i);
      if ((c & fixed) == prefix)
        atomicAdd(&hist256[(uint32_t)(c >> lo) & ((1u << width) - 1u)], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // 256 bins, 8 per lane
      const uint32_t lane = threadIdx.x;
      uint32_t own = 0;
      for (int i = 0; i < 8; i++) own += hist256[lane * 8 + i];
      uint32_t incl = own;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t u = __shfl_down_sync(0xFFFFFFFFu, incl, d);
        if (lane + d < 32) incl += u;
      }
      uint32_t excl = incl - own;
      bool mine = (excl < need_rem) && (incl >= need_rem);
      uint32_t msk = __ballot_sync(0xFFFFFFFFu, mine);
      uint32_t owner = msk ? (__ffs(msk) - 1) : 0;
      if (lane == owner) {
        uint32_t acc = excl;
        int bb = lane * 8 + 7;
        for (; bb > (int)(lane * 8); bb--) {
          if (acc + hist256[bb] >= need_rem) break;
          acc += hist256[bb];
        }
        sh64[66] = (uint64_t)bb;
        sh64[67] = (uint64_t)acc;
        sh64[68] = (uint64_t)hist256[bb];
      }
    }
    __syncthreads();
    const uint32_t d = (uint32_t)sh64[66];
    const uint32_t above = (uint32_t)sh64[67];
    const uint32_t inbin = (uint32_t)sh64[68];
    __syncthreads();
    need_rem -= above;
    prefix |= (uint64_t)d << lo;
    fixed |= (uint64_t)((1u << width) - 1u) << lo;
    if (inbin == need_rem || lo == 0) break;
    hi = lo - 1;
  }
  return prefix;
}

// ---------------------------------------------------------------------------------------------
// k_select: per (query, partition) exact Top-ntop of the survivors by (key desc, row desc), in any
// order.  implicit = true reads every row of the partition from a full key array (slow path).
//
// Latency-bound: some thousand survivors from L2 and a few block-wide steps.  One 2048-bin
// histogram of the keys puts all but the boundary bin's survivors on one side; those few are ranked
// by counting (6k survivors: 16 -> 8.4 us; the radix passes before took one 8-bit digit each).  Up
// to 16 survivors per thread stay in registers between the steps.  Where
// partitions keep few candidates each (k_select_warp), a warp per (query, partition) bounds the
// boundary by the maxima of 64 groups of its survivors instead and ranks those above.
// ---------------------------------------------------------------------------------------------
struct SelectArgs {
  const uint2* surv;        // [nq][split][cap]
  const uint32_t* cnt;      // [nq][split]
  uint32_t cap;
  const uint32_t* allkeys;  // implicit: [n_rows] keys of query `q0`
  uint32_t q0;
  uint32_t split, slice, n_rows, ntop;
  uint32_t* cand;           // [nq][split*ntop] rows, 0xFFFFFFFF = empty slot
  uint32_t* cand_key;       // [nq][split*ntop]
  uint32_t* status;         // [nq]
  uint32_t* done;           // [nq] (implicit: [1]) or null: k_final's CTA counters, zeroed here
  uint32_t pairs;           // k_select_warp: queries * split
};

constexpr int kThreadsSel = 512;
constexpr int kSelKeys = 16;             // survivors per thread kept in registers
constexpr uint32_t kSelListMax = 1024;   // survivors of the boundary bin ranked by counting

// Block-wide select of the `need` (1 <= need <= n) largest composites of the items key(i), row(i),
// i < n; each goes to put(slot, key, row), slots 0 .. need - 1 in any order.
template <int THREADS>
struct SelectShared {
  __align__(16) uint32_t hist[kHistBins];
  uint64_t sh64[72];
  uint64_t list[kSelListMax];
  uint32_t sh[THREADS / 32 + 3], wmin[THREADS / 32], wmax[THREADS / 32];
  uint32_t n_out, n_list;
};
template <int THREADS, bool REGS, class Key, class Row, class Put>
__device__ __forceinline__ void block_select(SelectShared<THREADS>& S, uint32_t n, uint32_t need,
                                             const Key& key, const Row& row, const Put& put) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t k[REGS ? kSelKeys : 1];
  if constexpr (REGS) {
#pragma unroll
    for (int u = 0; u < kSelKeys; u++) k[u] = u * THREADS + tid < n ? key(u * THREADS + tid) : 0u;
  }
  // f(item, its key) for this thread's items; every thread of a warp makes the same calls, with
  // item >= n for none
  auto each = [&](auto&& f) {
    if constexpr (REGS) {
#pragma unroll
      for (int u = 0; u < kSelKeys; u++)
        if (u * THREADS < n) f((uint32_t)(u * THREADS) + tid, k[u]);
    } else {
      for (uint32_t i0 = 0; i0 < n; i0 += THREADS * 4) {
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t i = i0 + u * THREADS + tid;
          v[u] = i < n ? key(i) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (i0 + u * THREADS < n) f(i0 + u * THREADS + tid, v[u]);
      }
    }
  };
  uint32_t mn = 0xFFFFFFFFu, mx = 0;
  each([&](uint32_t i, uint32_t v) {
    if (i < n) {
      mn = min(mn, v);
      mx = max(mx, v);
    }
  });
  mn = __reduce_min_sync(0xFFFFFFFFu, mn);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  if (lane == 0) {
    S.wmin[warp] = mn;
    S.wmax[warp] = mx;
  }
  if (tid == 0) S.n_out = S.n_list = 0;
  for (uint32_t i = tid; i < kHistBins; i += THREADS) S.hist[i] = 0;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < THREADS / 32; w++) {
    mn = min(mn, S.wmin[w]);
    mx = max(mx, S.wmax[w]);
  }
  const uint32_t span = mx - mn;
  const int bl = span ? 32 - __clz(span) : 0;
  const int shift = bl > 11 ? bl - 11 : 0;
  each([&](uint32_t i, uint32_t v) {
    if (i < n) atomicAdd(&S.hist[(v - mn) >> shift], 1u);
  });
  __syncthreads();
  TopBin t = block_top_bin<THREADS>(S.hist, need, S.sh);
  uint64_t tau = ~0ull;        // items of the boundary bin that are kept: composites >= tau
  const bool big = t.in > kSelListMax;
  if (big)                     // many equal or nearly equal keys: the exact boundary composite
    tau = block_select_tau([&](uint32_t i) -> uint64_t { return ((uint64_t)key(i) << 32) | row(i); },
                           n, need, S.hist, S.sh64);
  each([&](uint32_t i, uint32_t v) {
    const uint32_t bin = (v - mn) >> shift;
    bool take = i < n && bin > t.bin;
    uint32_t r = 0;
    if (take) r = row(i);
    if (i < n && bin == t.bin) {
      r = row(i);
      if (big) take = (((uint64_t)v << 32) | r) >= tau;
      else S.list[atomicAdd(&S.n_list, 1u)] = ((uint64_t)v << 32) | r;
    }
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, take);
    if (m) {
      uint32_t o = 0;
      if (lane == 0) o = atomicAdd(&S.n_out, (uint32_t)__popc(m));
      o = __shfl_sync(0xFFFFFFFFu, o, 0) + __popc(m & ((1u << lane) - 1u));
      if (take) put(o, v, r);
    }
  });
  __syncthreads();
  if (!big) {
    const uint32_t rest = need - t.above;  // of the boundary bin
    for (uint32_t i = tid; i < t.in; i += THREADS) {
      const uint64_t c = S.list[i];
      uint32_t above = 0;
      for (uint32_t j = 0; j < t.in; j++) above += S.list[j] > c ? 1u : 0u;
      if (above < rest) put(t.above + above, (uint32_t)(c >> 32), (uint32_t)c);
    }
  }
}

template <bool IMPLICIT>
__global__ void __launch_bounds__(kThreadsSel, 1) k_select(SelectArgs a) {
  grid_wait();
  grid_next();
  __shared__ SelectShared<kThreadsSel> S;
  const uint32_t p = blockIdx.x, q = IMPLICIT ? a.q0 : blockIdx.y;
  const uint32_t r0 = p * a.slice;
  const uint32_t r1 = (a.split <= 1 || p == a.split - 1) ? a.n_rows : (p + 1) * a.slice;
  const uint32_t prow = (a.split <= 1) ? a.n_rows : (r1 - r0);
  const uint32_t need = min(a.ntop, prow);
  uint32_t* cr = a.cand + ((size_t)q * a.split + p) * a.ntop;
  uint32_t* ck = a.cand_key + ((size_t)q * a.split + p) * a.ntop;
  if (a.done && p == 0 && threadIdx.x == 0) a.done[IMPLICIT ? 0u : q] = 0u;
  uint32_t n = IMPLICIT ? prow : a.cnt[(size_t)q * a.split + p];
  const bool over = !IMPLICIT && n > a.cap, miss = !IMPLICIT && n < need;
  for (uint32_t i = (over || miss ? 0u : need) + threadIdx.x; i < a.ntop; i += kThreadsSel) {
    cr[i] = 0xFFFFFFFFu;
    ck[i] = 0;
  }
  if (over || miss) {
    if (threadIdx.x == 0) atomicOr(a.status + q, over ? ST_OVERFLOW : ST_MISS);
    return;
  }
  if (need == 0) return;
  auto put = [&](uint32_t o, uint32_t key, uint32_t row) {
    cr[o] = row;
    ck[o] = key;
  };
  if constexpr (IMPLICIT) {
    const uint32_t base = (a.split <= 1) ? 0 : r0;
    block_select<kThreadsSel, false>(S, n, need, [&](uint32_t i) { return a.allkeys[base + i]; },
                                     [&](uint32_t i) { return base + i; }, put);
  } else {
    const uint2* sv = a.surv + ((size_t)q * a.split + p) * a.cap;
    auto key = [&](uint32_t i) { return sv[i].x; };
    auto row = [&](uint32_t i) { return sv[i].y; };
    if (n <= (uint32_t)(kThreadsSel * kSelKeys)) block_select<kThreadsSel, true>(S, n, need, key, row, put);
    else block_select<kThreadsSel, false>(S, n, need, key, row, put);
  }
}

// One warp per (query, partition), for partitions that keep few candidates: up to kSelWarpKeys
// survivors in registers, 32 per lane.  A pair with more, or with many keys at its boundary, is
// selected by the whole CTA afterwards.
constexpr uint32_t kSelWarpTop = 64;     // the most candidates per partition of this form
constexpr uint32_t kSelWarpKeys = 1024;
constexpr uint32_t kSelWarpList = 128;   // the most of them at or above the groups' bound
constexpr int kSelWarpThreads = 256;

__global__ void __launch_bounds__(kSelWarpThreads) k_select_warp(SelectArgs a) {
  grid_wait();
  grid_next();
  constexpr int N = kSelWarpKeys / 32, W = kSelWarpThreads / 32;
  __shared__ SelectShared<kSelWarpThreads> S;
  __shared__ uint64_t s_list[W][kSelWarpList];
  __shared__ uint32_t s_big[W];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  auto need_of = [&](uint32_t p) {
    const uint32_t r1 = (a.split <= 1 || p == a.split - 1) ? a.n_rows : (p + 1) * a.slice;
    return min(a.ntop, a.split <= 1 ? a.n_rows : r1 - p * a.slice);
  };
  const uint32_t i0 = blockIdx.x * W, pair = i0 + warp;
  bool big = false;
  if (pair < a.pairs) {
    const uint32_t p = pair % a.split, q = pair / a.split, need = need_of(p);
    if (a.done && p == 0 && lane == 0) a.done[q] = 0u;
    const uint32_t n = a.cnt[pair];
    uint32_t* cr = a.cand + (size_t)pair * a.ntop;
    uint32_t* ck = a.cand_key + (size_t)pair * a.ntop;
    const bool over = n > a.cap, miss = n < need;
    for (uint32_t i = (over || miss ? 0u : need) + lane; i < a.ntop; i += 32) {
      cr[i] = 0xFFFFFFFFu;
      ck[i] = 0;
    }
    if (over || miss) {
      if (lane == 0) atomicOr(a.status + q, over ? ST_OVERFLOW : ST_MISS);
    } else if (n > kSelWarpKeys) {
      big = need != 0;
    } else if (need) {
      const uint2* sv = a.surv + (size_t)pair * a.cap;
      uint32_t k[N], g[2] = {0u, 0u};  // the larger keys of two groups per lane
#pragma unroll
      for (int u = 0; u < N; u++) {
        const uint32_t i = u * 32 + lane;
        k[u] = i < n ? sv[i].x : 0u;
        g[u & 1] = max(g[u & 1], k[u]);
      }
      // the need-th largest of the 64 groups' maxima: need keys reach it and few others do
      const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, max(g[0], g[1]));
      const uint32_t mn = __reduce_min_sync(0xFFFFFFFFu, min(g[0], g[1]));
      const uint32_t t = warp_rth_key<2>(g, mn, mx, need);
      uint32_t own = 0;
#pragma unroll
      for (int u = 0; u < N; u++) own += (uint32_t)(u * 32) + lane < n && k[u] >= t ? 1u : 0u;
      const uint32_t incl = warp_incl_sum(own, lane);
      const uint32_t m = __shfl_sync(0xFFFFFFFFu, incl, 31);
      big = m > kSelWarpList;
      if (!big) {  // gather their places, then the rows in one go, and rank them by counting
        uint32_t o = incl - own;
#pragma unroll
        for (int u = 0; u < N; u++)
          if ((uint32_t)(u * 32) + lane < n && k[u] >= t) s_list[warp][o++] = u * 32 + lane;
        __syncwarp();
        for (uint32_t i = lane; i < m; i += 32) {
          const uint2 v = sv[s_list[warp][i]];
          s_list[warp][i] = ((uint64_t)v.x << 32) | v.y;
        }
        __syncwarp();
        for (uint32_t i = lane; i < m; i += 32) {
          const uint64_t c = s_list[warp][i];
          uint32_t x = 0;
          for (uint32_t j = 0; j < m; j++) x += s_list[warp][j] > c ? 1u : 0u;
          if (x < need) {
            cr[x] = (uint32_t)c;
            ck[x] = (uint32_t)(c >> 32);
          }
        }
      }
    }
  }
  if (lane == 0) s_big[warp] = big ? 1u : 0u;
  __syncthreads();
  for (int w = 0; w < W; w++) {
    if (!s_big[w]) continue;
    const uint32_t pr = i0 + w;
    const uint2* sv = a.surv + (size_t)pr * a.cap;
    uint32_t* cr = a.cand + (size_t)pr * a.ntop;
    uint32_t* ck = a.cand_key + (size_t)pr * a.ntop;
    block_select<kSelWarpThreads, false>(
        S, a.cnt[pr], need_of(pr % a.split), [&](uint32_t i) { return sv[i].x; },
        [&](uint32_t i) { return sv[i].y; },
        [&](uint32_t o, uint32_t key, uint32_t row) {
          cr[o] = row;
          ck[o] = key;
        });
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// k_final: FP32 rescoring of every candidate (sequential over the row's entries in column
// order, separately rounded multiply and add) and the final Top-K in sort_tuples order.
//
// Bound by latency: a candidate row is a dependent chain of the row pointer, then its entries,
// from DRAM.  So the candidates of a few queries are spread over gridDim.x CTAs of 16 warps each,
// and a warp takes 4 rows at a time: their entries are loaded row by row (lane = entry, coalesced;
// up to 128 per row in one round trip), the rounded products staged in shared memory, and lane r
// then sums row r's products in entry order.  The query's last CTA to finish selects the K best
// (score, row) composites.  With several hundred queries gridDim.x is 1, the composites stay in
// shared memory and, where there are rows for every warp, a warp takes 32 at a time, which costs
// a quarter of the summing steps.
// Selection: one 2048-bin histogram of the scores leaves K and a few more, which are ranked by
// counting (or, past 256, sorted).
// ---------------------------------------------------------------------------------------------
struct FinalArgs {
  const uint32_t* csr_ptr;   // [rows+1]
  const uint16_t* csr_col;
  const float* csr_val;
  const float* q32;          // [nq][ld32]
  uint32_t ld32, cols;
  const uint32_t* cand;      // [nq][nslots]
  uint32_t nslots, k;
  uint32_t* out_idx;         // [nq][k]
  float* out_score;          // [nq][k]
  const uint32_t* status;    // [nq]; queries with a set status are left to the repair path
  // [nq][nslots] candidate keys, or null.  Given: the final Top-K ranks the candidates by their
  // integer candidate score (no FP32 rescoring: a pre-quantised matrix or query without FP32
  // values) and out_score holds that score; with key_f32 they are the keys of FP32 scores that are
  // already exact
  const uint32_t* cand_key;
  uint32_t key_f32;
  uint32_t* status_out;      // [nq] or null: the status words, to pinned host memory
  uint64_t* comp;            // gridDim.x > 1: [nq][nslots] composites between the CTAs of a query
  uint32_t* done;            // gridDim.x > 1: [nq] CTAs finished, zero before the launch
};

constexpr int kThreadsFinal = 512;  // two CTAs per SM: a 256-query batch runs in one wave
constexpr int kFinalRows = 4;       // several CTAs per query: candidate rows a warp takes at a time
constexpr int kFinalChunk = 128;    // and entries per row staged at a time
constexpr int kFinalStage = 32 * 33;  // staged products per warp: 32 rows x 32 or 4 x 128, padded
static_assert(kFinalRows * (kFinalChunk + 1) <= kFinalStage, "staging");
constexpr uint32_t kFinalRankMax = 256;  // survivors of the histogram ranked by counting

// slots of the selected composites: K and what shares the K-th one's histogram bin
__host__ __device__ inline uint32_t final_list_slots(uint32_t k) {
  uint32_t n = 512;
  while (n < 2 * k) n <<= 1;
  return n;
}
// dynamic shared memory of k_final: the query, the composites of all slots, then one region
// holding first the per-warp product staging and afterwards the selected composites
__host__ __device__ inline size_t final_smem_bytes(uint32_t cols, uint32_t nslots, uint32_t k) {
  const size_t stage = (size_t)(kThreadsFinal / 32) * kFinalStage * 4;
  const size_t top = (size_t)final_list_slots(k) * 8;
  return (((size_t)cols * 4 + 15) & ~(size_t)15) + (size_t)nslots * 8 + (stage > top ? stage : top);
}

// FP32 scores of the candidate rows of one warp's group of ROWS: lane r < ROWS gets the score of
// its row (s: its first entry, n: its entries; 0 for the other lanes).  CHUNK entries of every row
// are staged at a time, the loads of several rows in flight.
template <int ROWS, int CHUNK>
__device__ __forceinline__ float rescore_rows(const FinalArgs& a, const float* qs, float* sp,
                                              uint32_t s, uint32_t n) {
  constexpr int U = CHUNK / 32, LD = CHUNK + 1;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t longest = __reduce_max_sync(0xFFFFFFFFu, n);
  float acc = 0.0f;
  for (uint32_t c = 0; c < longest; c += CHUNK) {
    if (U == 1 || longest - c <= 32u) {
#pragma unroll 8
      for (int j = 0; j < ROWS; j++) {
        const uint32_t sj = __shfl_sync(0xFFFFFFFFu, s, j), nj = __shfl_sync(0xFFFFFFFFu, n, j);
        const uint32_t o = c + lane;
        float p = 0.0f;
        if (o < nj) p = __fmul_rn(__ldg(a.csr_val + sj + o), qs[__ldg(a.csr_col + sj + o)]);
        sp[j * LD + lane] = p;
      }
    } else {
      constexpr int J = ROWS < 4 ? ROWS : 4;  // rows in flight
#pragma unroll 1
      for (int j0 = 0; j0 < ROWS; j0 += J) {
        float v[J][U];
        uint32_t cc[J][U];
#pragma unroll
        for (int j = 0; j < J; j++) {
          const uint32_t sj = __shfl_sync(0xFFFFFFFFu, s, j0 + j), nj = __shfl_sync(0xFFFFFFFFu, n, j0 + j);
#pragma unroll
          for (int u = 0; u < U; u++) {
            const uint32_t o = c + lane + 32u * u;
            v[j][u] = o < nj ? __ldg(a.csr_val + sj + o) : 0.0f;
            cc[j][u] = o < nj ? __ldg(a.csr_col + sj + o) : 0u;
          }
        }
#pragma unroll
        for (int j = 0; j < J; j++)
#pragma unroll
          for (int u = 0; u < U; u++)
            sp[(j0 + j) * LD + lane + 32 * u] = __fmul_rn(v[j][u], qs[cc[j][u]]);
      }
    }
    __syncwarp();
    const uint32_t m = n > c ? min(n - c, (uint32_t)CHUNK) : 0u;
    for (uint32_t e = 0; e < m; e++) acc = __fadd_rn(acc, sp[lane * LD + e]);
    __syncwarp();
  }
  return acc;
}

__global__ void __launch_bounds__(kThreadsFinal, 2) k_final(FinalArgs a) {
  grid_wait();
  grid_next();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) uint32_t hist[kHistBins];
  __shared__ uint64_t sh64[72];
  __shared__ uint32_t sh[kThreadsFinal / 32 + 3], swmin[kThreadsFinal / 32], swmax[kThreadsFinal / 32],
      swn[kThreadsFinal / 32];
  __shared__ uint32_t s_cnt, s_last;
  float* qs = reinterpret_cast<float*>(smem);
  uint64_t* comp = reinterpret_cast<uint64_t*>(smem + ((a.cols * 4 + 15) & ~15u));
  uint64_t* list = comp + a.nslots;  // after the rescoring; the product staging before it
  const uint32_t q = blockIdx.y;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (a.status) {
    const uint32_t st = a.status[q];
    if (a.status_out && blockIdx.x == 0 && threadIdx.x == 0) a.status_out[q] = st;
    if (st) return;
  }
  const uint32_t* cr = a.cand + (size_t)q * a.nslots;
  if (threadIdx.x == 0) s_cnt = 0;
  if (a.cand_key) {  // integer ranking: the candidate keys themselves (one CTA per query)
    const uint32_t* ck = a.cand_key + (size_t)q * a.nslots;
    for (uint32_t i = threadIdx.x; i < a.nslots; i += blockDim.x) {
      const uint32_t row = cr[i];
      comp[i] = row != 0xFFFFFFFFu ? ((uint64_t)ck[i] << 32) | row : 0ull;
    }
  } else {
    const float* x = a.q32 + (size_t)q * a.ld32;
    for (uint32_t j = threadIdx.x; j < a.cols; j += blockDim.x) qs[j] = x[j];
    __syncthreads();
    const bool many = gridDim.x > 1;
    const bool few = many || a.nslots < 32u * (kThreadsFinal / 32);  // a group of 32 leaves warps idle
    const uint32_t rows = few ? kFinalRows : 32u;
    float* sp = reinterpret_cast<float*>(list) + warp * kFinalStage;
    const uint32_t step = gridDim.x * (kThreadsFinal / 32) * rows;
    for (uint32_t g = (blockIdx.x * (kThreadsFinal / 32) + warp) * rows; g < a.nslots; g += step) {
      const uint32_t i = g + lane;
      const bool mine = lane < rows && i < a.nslots;
      const uint32_t row = mine ? cr[i] : 0xFFFFFFFFu;
      uint32_t s = 0, n = 0;
      if (row != 0xFFFFFFFFu) {
        s = __ldg(a.csr_ptr + row);
        n = __ldg(a.csr_ptr + row + 1) - s;
      }
      const float acc = few ? rescore_rows<kFinalRows, kFinalChunk>(a, qs, sp, s, n)
                            : rescore_rows<32, 32>(a, qs, sp, s, n);
      if (mine) {
        const uint64_t c = row != 0xFFFFFFFFu ? ((uint64_t)key_f32(acc) << 32) | row : 0ull;
        if (many) a.comp[(size_t)q * a.nslots + i] = c;
        else comp[i] = c;
      }
    }
    if (many) {  // the query's last CTA goes on with every CTA's composites
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) s_last = atomicAdd(a.done + q, 1u) == gridDim.x - 1;
      __syncthreads();
      if (!s_last) return;
      __threadfence();
      for (uint32_t i = threadIdx.x; i < a.nslots; i += blockDim.x)
        comp[i] = __ldcg(reinterpret_cast<const unsigned long long*>(a.comp) + (size_t)q * a.nslots + i);
    }
  }
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  // filled slots (composites of rows are unique and not 0; empty slots are 0), range of their keys
  uint32_t mn = 0xFFFFFFFFu, mx = 0, nv = 0;
  for (uint32_t i = threadIdx.x; i < a.nslots; i += blockDim.x) {
    const uint64_t c = comp[i];
    if (c != 0) {
      mn = min(mn, (uint32_t)(c >> 32));
      mx = max(mx, (uint32_t)(c >> 32));
      nv++;
    }
  }
  mn = __reduce_min_sync(0xFFFFFFFFu, mn);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  nv = __reduce_add_sync(0xFFFFFFFFu, nv);
  if (lane == 0) {
    swmin[warp] = mn;
    swmax[warp] = mx;
    swn[warp] = nv;
  }
  __syncthreads();
  nv = 0;
#pragma unroll
  for (int w = 0; w < kThreadsFinal / 32; w++) {
    mn = min(mn, swmin[w]);
    mx = max(mx, swmax[w]);
    nv += swn[w];
  }
  const uint32_t need = min(a.k, nv);
  uint32_t m = 0;
  if (need) {
    const uint32_t span = mx - mn;
    const int bl = span ? 32 - __clz(span) : 0;
    const int shift = bl > 11 ? bl - 11 : 0;
    for (uint32_t i = threadIdx.x; i < a.nslots; i += blockDim.x) {
      const uint64_t c = comp[i];
      if (c != 0) atomicAdd(&hist[((uint32_t)(c >> 32) - mn) >> shift], 1u);
    }
    __syncthreads();
    const TopBin t = block_top_bin<kThreadsFinal>(hist, need, sh);
    const uint32_t slots = final_list_slots(a.k);
    uint64_t tau = (uint64_t)(mn + (t.bin << shift)) << 32;
    m = t.above + t.in;
    if (m > slots) {  // many equal or nearly equal scores: the exact K-th composite
      tau = block_select_tau([&](uint32_t i) -> uint64_t { return comp[i]; }, a.nslots, need, hist, sh64);
      m = need;
    }
    for (uint32_t i = threadIdx.x; i < a.nslots; i += blockDim.x) {
      const uint64_t c = comp[i];
      if (c != 0 && c >= tau) list[atomicAdd(&s_cnt, 1u)] = c;
    }
    __syncthreads();
  }
  uint32_t* oi = a.out_idx + (size_t)q * a.k;
  float* os = a.out_score + (size_t)q * a.k;
  auto put = [&](uint32_t o, uint64_t c) {
    oi[o] = (uint32_t)c;
    const uint32_t key = (uint32_t)(c >> 32);
    os[o] = a.cand_key && !a.key_f32 ? (float)(int32_t)(key ^ 0x80000000u) : key_to_f32(key);
  };
  if (m <= kFinalRankMax) {
    // a composite's place is the number of larger ones, counted by `per` threads of a warp
    uint32_t per = 32;
    while (per > 1 && m * per > kThreadsFinal) per >>= 1;
    const uint32_t i = threadIdx.x / per, part = threadIdx.x % per;
    const uint64_t c = i < m ? list[i] : 0ull;
    uint32_t above = 0;
    if (i < m)
      for (uint32_t j = part; j < m; j += per) above += list[j] > c ? 1u : 0u;
    for (uint32_t d = per >> 1; d > 0; d >>= 1) above += __shfl_xor_sync(0xFFFFFFFFu, above, d);
    if (i < m && part == 0 && above < need) put(above, c);
  } else {  // bitonic sort, descending
    uint32_t np = 1;
    while (np < m) np <<= 1;
    for (uint32_t i = m + threadIdx.x; i < np; i += blockDim.x) list[i] = 0;
    __syncthreads();
    for (uint32_t kk = 2; kk <= np; kk <<= 1) {
      for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
        for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) {
          const uint32_t l = i ^ j;
          if (l > i) {
            const uint64_t ci = list[i], cl = list[l];
            const bool desc = ((i & kk) == 0);
            if (desc ? (ci < cl) : (ci > cl)) { list[i] = cl; list[l] = ci; }
          }
        }
        __syncthreads();
      }
    }
    for (uint32_t i = threadIdx.x; i < need; i += blockDim.x) put(i, list[i]);
  }
  for (uint32_t i = need + threadIdx.x; i < a.k; i += blockDim.x) {
    oi[i] = 0xFFFFFFFFu;
    os[i] = -__int_as_float(0x7f800000);
  }
}

}  // namespace dev
}  // namespace aes

namespace aes {
namespace dev {

// FP32-only pass: the FP32 score of every row (each row summed in column order with separately
// rounded multiply and add: spmv_coo_gold_top_k, gold_algorithms.hpp:189-247 with V = float) as an
// order-preserving key.  A warp takes 32 consecutive rows, one per lane.  Their entries are
// contiguous in the CSR, so the warp walks them in chunks of kExactChunk: every lane loads entries
// of the chunk (coalesced, all loads in flight at once) and stores their rounded products
// v * q[col] to shared memory in entry order; then each lane adds its own row's products of the
// chunk in order.  The products and the order of the additions are those of the sequential sum.
constexpr uint32_t kExactChunk = 512;       // entries per warp and chunk
constexpr uint32_t kExactWarps = 8;         // warps per CTA
__host__ inline size_t exact_all_smem_bytes(uint32_t cols) {
  return (size_t)cols * 4 + (size_t)kExactWarps * kExactChunk * 4;
}

// FILTER: no keys array; rows at or above the threshold go to the survivors (the count goes on past
// cap, so that the select can tell an overflow).
template <bool FILTER>
__global__ void __launch_bounds__(kExactWarps * 32) k_exact_all(
    const uint32_t* __restrict__ ptr, const uint16_t* __restrict__ col,
    const float* __restrict__ val, const float* __restrict__ q, uint32_t cols, uint32_t rows,
    uint32_t* __restrict__ keys, const uint32_t* thr, uint32_t* __restrict__ cnt,
    uint2* __restrict__ surv, uint32_t cap) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char xsm[];
  float* qs = reinterpret_cast<float*>(xsm);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  float* sp = reinterpret_cast<float*>(xsm + (size_t)cols * 4) + warp * kExactChunk;
  for (uint32_t j = threadIdx.x; j < cols; j += blockDim.x) qs[j] = q[j];
  const uint32_t th = FILTER ? *thr : 0u;
  __syncthreads();
  const uint32_t nblk = (rows + 31) / 32;
  for (uint32_t blk = blockIdx.x * kExactWarps + warp; blk < nblk; blk += gridDim.x * kExactWarps) {
    const uint32_t r0 = blk * 32, r = r0 + lane;
    const uint32_t rend = min(r0 + 32u, rows);
    const uint32_t E0 = ptr[r0], E1 = ptr[rend];
    const uint32_t s = r < rows ? ptr[r] : E1, e = r < rows ? ptr[r + 1] : E1;
    float acc = 0.0f;
    for (uint32_t c = E0; c < E1; c += kExactChunk) {
      const uint32_t n = min(kExactChunk, E1 - c);
      float lv[kExactChunk / 32];
      uint32_t lc[kExactChunk / 32];
#pragma unroll
      for (uint32_t u = 0; u < kExactChunk / 32; u++) {
        const uint32_t i = u * 32 + lane;
        lv[u] = i < n ? __ldcs(val + c + i) : 0.0f;
        lc[u] = i < n ? (uint32_t)__ldcs(col + c + i) : 0u;
      }
#pragma unroll
      for (uint32_t u = 0; u < kExactChunk / 32; u++) sp[u * 32 + lane] = __fmul_rn(lv[u], qs[lc[u]]);
      __syncwarp();
      const uint32_t a = max(s, c), b = min(e, c + n);
      for (uint32_t i = a; i < b; i++) acc = __fadd_rn(acc, sp[i - c]);
      __syncwarp();
    }
    if (r < rows) {
      const uint32_t key = key_f32(acc);
      if constexpr (FILTER) {
        if (key >= th) {
          const uint32_t i = atomicAdd(cnt, 1u);
          if (i < cap) surv[i] = make_uint2(key, r);
        }
      } else {
        keys[r] = key;
      }
    }
  }
}

// FP32-only pass with a bound: rows whose key is at least their query's threshold are appended to
// its survivors; nothing is written for the others.  T queries per matrix read.
struct ExactArgs {
  const uint32_t* ptr;
  const uint16_t* col;
  const float* val;
  const float* q;       // [nq][ld], the launch's first query
  uint32_t ld, cols, rows, nq;
  const uint32_t* thr;  // [nq]
  uint32_t* cnt;        // [nq]; counts on past cap, so that the select can tell an overflow
  uint2* surv;          // [nq][cap]
  uint32_t cap;
};

// Bound by shared memory: an entry gathers T queries' values of its column.  T / 4 lanes walk a row
// in column order, four queries each, so the 16-byte loads of eight lanes cover 32 / T rows' columns;
// the table keeps a column's T values 32 / T times side by side, 128 bytes in all, and each of the
// rows reads its own copy: no two lanes meet in a bank whatever the columns (one copy with a lane
// per row, two loads for eight queries: 2.7 wavefronts instead of one per eight lanes).  A warp
// stages its 128 / T rows' entries (contiguous in the CSR) in chunks, the next chunk's loads under
// way while it walks.  1M rows x 20 entries, 16 queries: 205 -> 106 us.  blockIdx.y: the group of T
// queries.
// Two forms: 32 warps with 256 staged entries each, or 16 with 512 (LONG) where a warp's rows have more
// than 256 on average (exact_multi_long): eight queries, 16 rows to a warp, 1M x 20 127 / 112 us,
// 3M x 8.5 130 / 163 us; 16 queries, 8 rows to a warp, 1M x 20 151 / 162 us, 1M x 40 289 / 222 us.
template <int T, bool LONG>
struct ExMulti {
  static constexpr uint32_t WARPS = LONG ? 16 : 32;
  static constexpr uint32_t CHUNK = LONG ? 512 : 256;  // entries per warp and chunk
  static constexpr uint32_t HITS = 64;  // hits a warp collects before it appends them, 32 at a time or more
  __host__ static size_t smem(uint32_t cols) {
    return (size_t)cols * 128 + (size_t)WARPS * (CHUNK * 8 + HITS * 12);
  }
};
template <int T>
__host__ inline bool exact_multi_long(uint64_t nnz, uint32_t rows) {
  return nnz * (128 / T) > 256ull * rows;
}
template <int T, bool LONG>
__global__ void __launch_bounds__(ExMulti<T, LONG>::WARPS * 32, 1) k_exact_multi(ExactArgs a) {
  static_assert(T == 4 || T == 8 || T == 16, "queries per walk");
  constexpr uint32_t kWarps = ExMulti<T, LONG>::WARPS, kChunk = ExMulti<T, LONG>::CHUNK;
  constexpr uint32_t kHits = ExMulti<T, LONG>::HITS;
  constexpr uint32_t L = T / 4, R = 32 / L, COPIES = 32 / T, U = kChunk / 32;
  extern __shared__ __align__(128) unsigned char xsm[];
  float* qs = reinterpret_cast<float*>(xsm);  // [cols][COPIES][T]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  uint2* st = reinterpret_cast<uint2*>(xsm + (size_t)a.cols * 128) + warp * kChunk;
  // hits {query, key, row}: one atomic round trip for 32 of them, not one for each block of rows with a
  // hit (100k rows, 64 queries, the whole call: 352 -> 192 us)
  uint32_t* hits = reinterpret_cast<uint32_t*>(xsm + (size_t)a.cols * 128 + (size_t)kWarps * kChunk * 8) +
                   warp * kHits * 3;
  uint32_t nh = 0;
  auto flush = [&]() {
    __syncwarp();
    for (uint32_t i = lane; i < nh; i += 32) {
      const uint32_t q = hits[i], at = atomicAdd(a.cnt + q, 1u);
      if (at < a.cap)
        a.surv[(size_t)q * a.cap + at] = make_uint2(hits[kHits + i], hits[2 * kHits + i]);
    }
    __syncwarp();
    nh = 0;
  };
  const uint32_t q0 = blockIdx.y * T, nq = min((uint32_t)T, a.nq - q0);
  {  // a thread takes one query's value of every COPIES-th group of columns; writes without conflicts
    const uint32_t t = lane % T, sub = lane / T;
    const float* x = a.q + (size_t)(q0 + min(t, nq - 1u)) * a.ld;
#pragma unroll 8
    for (uint32_t j = warp * COPIES + sub; j < a.cols; j += kWarps * COPIES) {
      const float v = x[j];
#pragma unroll
      for (uint32_t k = 0; k < COPIES; k++) qs[j * 32u + (sub + k) % COPIES * T + t] = v;
    }
  }
  const uint32_t g = lane / L, l = lane % L;
  uint32_t th[4];
#pragma unroll
  for (uint32_t t = 0; t < 4; t++) th[t] = 4 * l + t < nq ? a.thr[q0 + 4 * l + t] : 0xFFFFFFFFu;
  const unsigned char* mine = xsm + lane % 8u * 16u;  // the row's copy, this lane's queries
  __syncthreads();
  const uint32_t nblk = (a.rows + R - 1) / R, stride = gridDim.x * kWarps;
  // this lane's row of block blk (past the matrix: empty)
  auto bounds = [&](uint64_t blk, uint32_t& s, uint32_t& e) {
    const uint64_t r = blk * R + g;
    s = a.ptr[min(r, (uint64_t)a.rows)];
    e = a.ptr[min(r + 1, (uint64_t)a.rows)];
  };
  float lv[U];
  uint32_t lc[U];
  auto load = [&](uint32_t c, uint32_t E1) {
    const uint32_t n = min(kChunk, E1 - c);
#pragma unroll
    for (uint32_t u = 0; u < U; u++) {
      const uint32_t i = u * 32 + lane;
      lv[u] = i < n ? __ldg(a.val + c + i) : 0.0f;
      lc[u] = i < n ? (uint32_t)__ldg(a.col + c + i) : 0u;
    }
  };
  uint32_t blk = warp * gridDim.x + blockIdx.x;  // (a small matrix spreads over the CTAs)
  uint32_t s, e, sn, en;
  bounds(blk, s, e);
  bounds((uint64_t)blk + stride, sn, en);
  uint32_t c = __shfl_sync(0xFFFFFFFFu, s, 0), E1 = __shfl_sync(0xFFFFFFFFu, e, 31);
  load(c, E1);
  while (blk < nblk) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (bool more = true; more;) {
      const uint32_t n = min(kChunk, E1 - c), c0 = c, e0 = c + n;
      __syncwarp();
#pragma unroll
      for (uint32_t u = 0; u < U; u++)
        if (u * 32 < n) st[u * 32 + lane] = make_uint2(__float_as_uint(lv[u]), lc[u] * 128u);
      __syncwarp();
      more = E1 - c > kChunk;
      if (more) {
        c += kChunk;
      } else {
        c = __shfl_sync(0xFFFFFFFFu, sn, 0);
        E1 = __shfl_sync(0xFFFFFFFFu, en, 31);
      }
      load(c, E1);
      const uint32_t d = min(e, e0);
#pragma unroll 4
      for (uint32_t i = max(s, c0); i < d; i++) {
        const uint2 w = st[i - c0];
        const float v = __uint_as_float(w.x);
        const float4 x = *reinterpret_cast<const float4*>(mine + w.y);
        acc[0] = __fadd_rn(acc[0], __fmul_rn(v, x.x));
        acc[1] = __fadd_rn(acc[1], __fmul_rn(v, x.y));
        acc[2] = __fadd_rn(acc[2], __fmul_rn(v, x.z));
        acc[3] = __fadd_rn(acc[3], __fmul_rn(v, x.w));
      }
    }
    const uint32_t r = blk * R + g;
#pragma unroll
    for (uint32_t t = 0; t < 4; t++) {
      const uint32_t key = key_f32(acc[t]);
      const bool hit = key >= th[t] && r < a.rows && 4 * l + t < nq;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
      if (!m) continue;
      if (nh + __popc(m) > kHits) flush();
      if (hit) {
        const uint32_t at = nh + __popc(m & ((1u << lane) - 1u));
        hits[at] = q0 + 4 * l + t;
        hits[kHits + at] = key;
        hits[2 * kHits + at] = r;
      }
      nh += __popc(m);
    }
    s = sn;
    e = en;
    if (nblk - blk <= stride) break;
    blk += stride;
    bounds((uint64_t)blk + stride, sn, en);
  }
  flush();
}

// One CTA per SM, shared out over g groups of T queries
template <int T>
__host__ inline void launch_exact_multi(const ExactArgs& x, uint32_t g, uint64_t nnz, int sm_count, cudaStream_t s) {
  const dim3 grid(std::max<uint32_t>(1, (uint32_t)sm_count / g), g);
  if (exact_multi_long<T>(nnz, x.rows))
    k_exact_multi<T, true><<<grid, ExMulti<T, true>::WARPS * 32, ExMulti<T, true>::smem(x.cols), s>>>(x);
  else
    k_exact_multi<T, false><<<grid, ExMulti<T, false>::WARPS * 32, ExMulti<T, false>::smem(x.cols), s>>>(x);
}

// FP32 keys of rows 0, S, 2 S, ... (ns of them) per query (blockIdx.y): keys[nq][ns].  A warp takes
// 8 sampled rows: latency-bound, their entries in one round trip.
constexpr int kThreadsExSample = 256;
constexpr uint32_t kExSampleRows = kThreadsExSample / 32 * 8;  // per CTA
__host__ inline size_t exact_sample_smem_bytes(uint32_t cols) {
  return (((size_t)cols * 4 + 15) & ~(size_t)15) + (size_t)(kThreadsExSample / 32) * kFinalStage * 4;
}
__global__ void __launch_bounds__(kThreadsExSample) k_exact_sample(FinalArgs a, uint32_t S, uint32_t ns,
                                                                   uint32_t* __restrict__ keys) {
  grid_wait();
  grid_next();
  extern __shared__ __align__(16) unsigned char xsm[];
  float* qs = reinterpret_cast<float*>(xsm);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  float* sp = reinterpret_cast<float*>(xsm + ((a.cols * 4 + 15) & ~15u)) + warp * kFinalStage;
  const float* x = a.q32 + (size_t)blockIdx.y * a.ld32;
  for (uint32_t j = threadIdx.x; j < a.cols; j += blockDim.x) qs[j] = x[j];
  __syncthreads();
  for (uint32_t g = (blockIdx.x * (kThreadsExSample / 32) + warp) * 8; g < ns;
       g += gridDim.x * kExSampleRows) {
    const uint32_t i = lane < 8 ? g + lane : ns;
    uint32_t s = 0, n = 0;
    if (i < ns) {
      s = __ldg(a.csr_ptr + (size_t)i * S);
      n = __ldg(a.csr_ptr + (size_t)i * S + 1) - s;
    }
    const float acc = rescore_rows<8, 32>(a, qs, sp, s, n);
    if (i < ns) keys[(size_t)blockIdx.y * ns + i] = key_f32(acc);
  }
}

}  // namespace dev
}  // namespace aes
