// aes_tf.cuh -- the tensor-core pass as a filter for values that FP8 does not hold exactly: the
// matrix and query preparation around k_cand_tc, and the exact check of what it lets through.
//
// A row score s = sum v q of 6- or 8-bit integers is approximated by s' = sum v' q', the products
// of the nearest e4m3 values v' of v and q' of q - c (c: one centre for the launch's queries, which
// halves the largest rounding error of a one-sided query).  With d = v - v' and e = (q - c) - q',
//     s = s' + c sum v + sum v' e + sum d (q - c),
// so |s - s' - c sum v| <= E sum |v'| + Q sum |d|, with E = max |e| and Q = max |q - c| over the
// launch's queries.  Per row, sum v, sum |v'| and sum |d| are known beforehand; the pass keeps
// every (row, query) whose s' plus this bound reaches the threshold, 1 to 2.6 times the rows that
// reach it themselves (uniform and normal values, dense and signed queries), and k_recheck scores
// those exactly in integers and drops the rest.  What is left is what the dp4a pass
// (aes_batch.cuh) leaves, at the FP8 rate of the tensor cores instead of the dp4a issue rate.
#pragma once

#include <algorithm>

#include "aes_select.cuh"
#include "aes_tc.cuh"

namespace aes {
namespace dev {

// nearest e4m3 integer of |v| <= 255 (ties to even): 4 significant bits
__device__ __forceinline__ int tf_round(int v) {
  const uint32_t m = (uint32_t)(v < 0 ? -v : v);
  if (m <= 16u) return v;
  const int s = 28 - __clz(m);  // bits dropped
  uint32_t k = m >> s;
  const uint32_t rem = m & ((1u << s) - 1u), half = 1u << (s - 1);
  if (rem > half || (rem == half && (k & 1u))) k++;
  const int r = (int)(k << s);
  return v < 0 ? -r : r;
}
// its e4m3 byte
__device__ __forceinline__ uint32_t tf_byte(int r) {
  if (r == 0) return 0u;
  const uint32_t m = (uint32_t)(r < 0 ? -r : r);
  const int e = 31 - __clz(m);
  return (r < 0 ? 0x80u : 0u) | (uint32_t)(e + 7) << 3 | ((m << 3 >> e) & 7u);
}

// Quantised rows, entry i of row r at 4 * tf_row4(ptr[r], r) + i: every row starts on 16 bytes and is
// padded with zeros (the rows' places do not overlap: ceil(n / 4) <= floor(n / 4) + 1)
__host__ __device__ inline uint64_t tf_row4(uint32_t first, uint32_t row) {
  return (uint64_t)(first >> 2) + row;
}
__host__ inline size_t tf_row_words(uint64_t nnz, uint32_t rows) { return 4 * (size_t)(nnz / 4 + rows + 1); }

__host__ __device__ inline uint64_t tf_mix(uint64_t x) {  // splitmix64, as the packer's empty-row rule
  uint64_t z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// ---- matrix side, once per matrix --------------------------------------------------------------
struct TfMatrix {
  const uint32_t* ptr;  // FP32 CSR
  const uint16_t* col;
  const float* val;
  uint32_t rows, cols, nch;
  int bits, quant;      // quantiser of the matrix
  float gmax;           // max |v| of the matrix (global quantisers)
  uint32_t* q;          // quantised rows (tf_row4): value << 16 | column
  uint2* rowstat;       // [rows] {sum |v'| << 13 | ceil(sum |d| / 2), sum v}
  uint32_t* ent;        // tensor-core layout (aes_tc.cuh): [nnz]
  uint32_t* tptr;       // [row tiles * nch + 1]
};

// A warp per row: the values quantised as the packer does (quantize_and_pack: the float64 arithmetic
// in integers, the empty-row rule) and the row's sums.  A row without entries scores the query at
// its seeded column: no entry here, so all of it is in the bound (d = 1).
__global__ void __launch_bounds__(256) k_tf_rows(TfMatrix a) {
  const uint32_t lane = threadIdx.x & 31u;
  const int32_t M = a.quant == 0 ? ((1 << a.bits) - 1) / 2 : (1 << a.bits) - 1;
  const int32_t lo = a.quant == 0 ? -M - 1 : 0;
  for (uint32_t r = blockIdx.x * 8 + (threadIdx.x >> 5); r < a.rows; r += gridDim.x * 8) {
    const uint32_t s = a.ptr[r], e = a.ptr[r + 1];
    // the row's largest value and its first place: the per-row scale, and where the empty-row rule
    // puts its entry (non-negative FP32 values order as their bits)
    uint32_t big = 0, at = 0xFFFFFFFFu;
    for (uint32_t i = s + lane; i < e; i += 32) {
      const uint32_t b = __float_as_uint(fabsf(a.val[i]));
      if (at == 0xFFFFFFFFu || b > big) {
        big = b;
        at = i;
      }
    }
    const uint32_t top = __reduce_max_sync(0xFFFFFFFFu, big);
    at = __reduce_min_sync(0xFFFFFFFFu, big == top ? at : 0xFFFFFFFFu);
    const float m = a.quant == 1 ? __uint_as_float(top) : a.gmax;
    uint32_t r1 = 0, r2 = 0, any = 0;
    int32_t rs = 0;
    for (uint32_t i0 = s; i0 < e; i0 += 32) {
      const uint32_t i = i0 + lane;
      if (i < e) {
        int32_t q = m != 0.0f ? qx::round_scaled(a.val[i], m, M) : 0;
        q = q < lo ? lo : (q > M ? M : q);
        const int v = tf_round(q);
        a.q[4 * tf_row4(s, r) + (i - s)] = (uint32_t)q << 16 | a.col[i];
        any |= q != 0;
        r1 += (uint32_t)(v < 0 ? -v : v);
        r2 += (uint32_t)(q > v ? q - v : v - q);
        rs += q;
      }
    }
    if (!__any_sync(0xFFFFFFFFu, any)) {  // a row left empty gets one entry
      __syncwarp();  // (after the zero that another lane stored in its place: a vote orders no memory)
      if (s == e) {
        r2 = lane == 0;
        rs = lane == 0;
      } else if (lane == 0) {
        const int32_t q = a.quant == 0 && a.val[at] < 0.0f ? -1 : 1;
        a.q[4 * tf_row4(s, r) + (at - s)] = (uint32_t)q << 16 | a.col[at];
        r1 = 1;
        rs = q;
      }
    }
    r1 = __reduce_add_sync(0xFFFFFFFFu, r1);
    r2 = __reduce_add_sync(0xFFFFFFFFu, r2);
    rs = __reduce_add_sync(0xFFFFFFFFu, rs);
    if (lane == 0) a.rowstat[r] = make_uint2(r1 << 13 | (r2 + 1) >> 1, (uint32_t)rs);
  }
}

// A CTA per 128-row tile: its entries grouped by 256-column chunk (the tile's are contiguous in the
// CSR, and stay in that range), each its operand offset << 16 | its e4m3 byte
__global__ void __launch_bounds__(256) k_tf_tiles(TfMatrix a) {
  __shared__ uint32_t n[4], pos[4];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t tiles = (a.rows + kTcRows - 1) / kTcRows;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint32_t r0 = t * kTcRows, r1 = min(r0 + kTcRows, a.rows);
    if (threadIdx.x < 4) n[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t i = a.ptr[r0] + threadIdx.x; i < a.ptr[r1]; i += 256) atomicAdd(&n[a.col[i] >> 8], 1u);
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t o = a.ptr[r0];
      for (uint32_t c = 0; c < a.nch; c++) {
        pos[c] = o;
        a.tptr[(size_t)t * a.nch + c] = o;
        o += n[c];
      }
      if (t == tiles - 1) a.tptr[(size_t)tiles * a.nch] = o;
    }
    __syncthreads();
    for (uint32_t r = r0 + warp; r < r1; r += 8) {
      const uint32_t s = a.ptr[r], e = a.ptr[r + 1];
      for (uint32_t i0 = s; i0 < e; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t c = i < e ? a.col[i] : 0xFFFFu;
        for (uint32_t k = 0; k < a.nch; k++) {
          const uint32_t mk = __ballot_sync(0xFFFFFFFFu, (c >> 8) == k);
          if (!mk) continue;
          uint32_t o = 0;
          if (lane == 0) o = atomicAdd(&pos[k], (uint32_t)__popc(mk));
          o = __shfl_sync(0xFFFFFFFFu, o, 0) + __popc(mk & ((1u << lane) - 1u));
          if ((c >> 8) == k) {
            const int q = (int)a.q[4 * tf_row4(s, r) + (i - s)] >> 16;
            a.ent[o] = tc_off(r - r0, c & 255u) << 16 | tf_byte(tf_round(q));
          }
        }
      }
    }
    __syncthreads();
  }
}

// ---- queries -----------------------------------------------------------------------------------
// Words of one launch's query statistics, zero before k_tf_qstats: max(512 + q), max(512 - q) over
// every query value, then E and Q.
constexpr uint32_t kTfStats = 4;

__global__ void __launch_bounds__(256) k_tf_qstats(const int8_t* q8, uint32_t ld8,
                                                   uint32_t cols, uint32_t sgn, uint32_t* st) {
  grid_wait();
  grid_next();
  uint32_t hi = 0, lo = 0;
  for (uint32_t c = threadIdx.x; c < cols; c += 256) {
    const int8_t b = q8[(size_t)blockIdx.x * ld8 + c];
    const int q = sgn ? (int)b : (int)(uint8_t)b;
    hi = max(hi, (uint32_t)(512 + q));
    lo = max(lo, (uint32_t)(512 - q));
  }
  hi = __reduce_max_sync(0xFFFFFFFFu, hi);
  lo = __reduce_max_sync(0xFFFFFFFFu, lo);
  if ((threadIdx.x & 31u) == 0) {
    atomicMax(st, hi);
    atomicMax(st + 1, lo);
  }
}

// e4m3 operands of every 128-query block, and E and Q.  A thread takes 16 columns of a query, 16
// bytes of both layouts (rows of q8 are padded to 16, and the operand's k 16 j .. 16 j + 15 of one
// query are contiguous).
__global__ void __launch_bounds__(256) k_tf_qtable(const int8_t* q8, uint32_t ld8,
                                                   uint32_t cols, uint32_t nq, uint32_t nblk, uint32_t sgn,
                                                   uint32_t* st, uint8_t* __restrict__ qt) {
  grid_wait();
  grid_next();
  const uint32_t per = tc_kpad(cols) / 16u;
  const int centre = tc_centre(st);
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  const uint32_t n = i / per, k0 = i % per * 16u;  // query of the batch, padded to whole blocks
  uint32_t E = 0, Q = 0;
  if (n < nblk * kTcQ) {
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (n < nq && k0 < cols) {
      const uint4 v = *reinterpret_cast<const uint4*>(q8 + (size_t)n * ld8 + k0);
      const uint32_t in[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint32_t b = in[j / 4] >> (8 * (j % 4)) & 255u;
        const int q = (sgn ? (int)(int8_t)b : (int)b) - centre;
        if (k0 + j < cols) {
          const int r = tf_round(q);
          w[j / 4] |= tf_byte(r) << (8 * (j % 4));
          E = max(E, (uint32_t)(q > r ? q - r : r - q));
          Q = max(Q, (uint32_t)(q < 0 ? -q : q));
        }
      }
    }
    *reinterpret_cast<uint4*>(qt + (size_t)(n / kTcQ) * tc_qtab_bytes(cols) + tc_off(n % kTcQ, k0)) =
        make_uint4(w[0], w[1], w[2], w[3]);
  }
  E = __reduce_max_sync(0xFFFFFFFFu, E);
  Q = __reduce_max_sync(0xFFFFFFFFu, Q);
  if ((threadIdx.x & 31u) == 0) {
    if (E) atomicMax(st + 2, E);
    if (Q) atomicMax(st + 3, Q);
  }
}

// ---- the exact check ---------------------------------------------------------------------------
struct TfCheck {
  const uint32_t* ptr;
  const uint4* q;         // quantised rows (tf_row4)
  uint32_t cols;
  uint64_t seed;          // of the empty-row rule
  const int8_t* q8;       // [nq_total][ld8]
  uint32_t ld8, sgn;
  uint32_t q0, nq;        // the filter launch's queries q0 .. q0 + nq - 1
  const uint2* list;      // [ctas][kTcLists][list_cap] {row, mask of the block's 32 queries}
  const uint32_t* list_n; // [ctas][kTcLists]
  uint32_t list_cap, ctas;
  const float* rowscale;
  const uint32_t* thr;    // [nq_total][split]
  uint32_t split, slice, cap;
  uint32_t* status;       // [nq_total]
  uint32_t* cnt;          // [nq_total][split]
  uint2* surv;            // [nq_total][split][cap]
};

constexpr int kThreadsCheck = 256;
// groups of eight rows whose first loads are in flight together (1: 40 registers and not 80, twice the
// warps; 512 queries on 4M x 1024 1558 us for 1541, 100 on 400k x 500 200 for 196)
constexpr int kCheckRows = 4;
// bytes per query in shared memory: a word more than the row, so that the bytes of several queries at
// one column (hits of one row) lie in different banks
__host__ __device__ inline uint32_t check_ld(uint32_t ld8) { return ld8 + 4u; }
__host__ inline size_t check_smem_bytes(uint32_t ld8) { return (size_t)check_ld(ld8) * 32; }

// What a filter launch let through for block blockIdx.x of 32 queries: every (row, query) is scored
// exactly and, at or above the threshold, appended to the query's survivors.  The block's queries
// sit in shared memory; the CTAs of a block share the lists of the filter's CTAs, a
// warp takes 32 list entries and spreads their hits over its lanes (a mask may hold one or 32).
// Bound by L2 and instruction issue: four lanes take a row, each 16 bytes (four entries) at a time,
// so a warp reads eight rows' 64-byte pieces per load and an entry costs four instructions, among
// them the gather of the query's byte.
__global__ void __launch_bounds__(kThreadsCheck) k_recheck(TfCheck a) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char csm[];
  __shared__ uint32_t s_most;  // entries of the longest list
  const int8_t* qs = reinterpret_cast<const int8_t*>(csm);
  const uint32_t ld = check_ld(a.ld8);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t blk = blockIdx.x, qb = a.q0 + blk * 32u, nb = min(32u, a.nq - blk * 32u);
  for (uint32_t q = warp; q < nb; q += kThreadsCheck / 32) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(a.q8 + (size_t)(qb + q) * a.ld8);
    for (uint32_t i = lane; i < a.ld8 / 4u; i += 32)
      reinterpret_cast<uint32_t*>(csm + q * ld)[i] = src[i];
  }
  if (threadIdx.x == 0) s_most = 0;
  __syncthreads();
  for (uint32_t l = threadIdx.x; l < a.ctas; l += kThreadsCheck) atomicMax(&s_most, a.list_n[l * kTcLists + blk]);
  __syncthreads();
  if (s_most > a.list_cap) {
    if (threadIdx.x < nb && blockIdx.y == 0) atomicOr(a.status + qb + threadIdx.x, ST_LIST);
    return;
  }
  // pieces of 32 entries, the j-th of every list before the next, over all warps of the block's CTAs
  const uint32_t pieces = (s_most + 31u) / 32u * a.ctas;
  for (uint32_t id = blockIdx.y * (kThreadsCheck / 32) + warp; id < pieces;
       id += gridDim.y * (kThreadsCheck / 32)) {
    const uint32_t l = id % a.ctas;
    const uint32_t n = a.list_n[l * kTcLists + blk];
    const uint2* list = a.list + ((size_t)l * kTcLists + blk) * a.list_cap;
    const uint32_t ei = id / a.ctas * 32u + lane;
    if (ei - lane >= n) continue;
    const uint2 ent = ei < n ? list[ei] : make_uint2(0u, 0u);
    uint32_t s = 0, m = 0;
    if (ei < n) {
      s = __ldg(a.ptr + ent.x);
      m = __ldg(a.ptr + ent.x + 1) - s;
    }
    const uint64_t at = tf_row4(s, ent.x);
    const uint32_t incl = warp_incl_sum(__popc(ent.y), lane);
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    for (uint32_t h0 = 0; h0 < total; h0 += 32u) {
      const uint32_t h = h0 + lane;
      uint32_t q = 0;
      uint32_t e = 0;  // the entry of hit h: how many of the inclusive sums are <= h
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, incl, e + d - 1) <= h) e += d;
      const uint32_t mk = __shfl_sync(0xFFFFFFFFu, ent.y, e);
      uint32_t k = h - (__shfl_sync(0xFFFFFFFFu, incl, e) - __popc(mk));  // its k-th set bit
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        const uint32_t c = __popc((mk >> q) & ((1u << d) - 1u));
        if (c <= k) {
          k -= c;
          q += d;
        }
      }
      const uint32_t row = __shfl_sync(0xFFFFFFFFu, ent.x, e);
      const uint32_t n4 = (__shfl_sync(0xFFFFFFFFu, m, e) + 3u) >> 2;
      const uint64_t src_h = __shfl_sync(0xFFFFFFFFu, at, e);
      const size_t qp = (size_t)(qb + q) * a.split + part_of(row, a.split, a.slice);
      const uint32_t th = h < total ? __ldg(a.thr + qp) : 0xFFFFFFFFu;  // (not a dependent launch)
      int32_t score = 0;
      if (h < total && n4 == 0) {
        const uint32_t c = (uint32_t)(tf_mix(a.seed ^ (uint64_t)row) % (uint64_t)a.cols);
        score = a.sgn ? (int)qs[q * ld + c] : (int)csm[q * ld + c];
      }
#pragma unroll
      for (int j0 = 0; j0 < 32; j0 += 8 * kCheckRows) {
        if (h0 + j0 >= total) break;
        // the first 32 entries of each row in flight together
        uint32_t nj[kCheckRows];
        const uint4* src[kCheckRows];
        uint4 x0[kCheckRows], x1[kCheckRows];
#pragma unroll
        for (int w = 0; w < kCheckRows; w++) {
          const int j = j0 + 8 * w + (int)(lane >> 2);
          const uint32_t n4j = __shfl_sync(0xFFFFFFFFu, n4, j);
          nj[w] = h0 + j < total ? n4j : 0u;
          src[w] = a.q + __shfl_sync(0xFFFFFFFFu, src_h, j);
          const uint32_t k4 = lane & 3u;
          x0[w] = k4 < nj[w] ? __ldg(src[w] + k4) : make_uint4(0u, 0u, 0u, 0u);
          x1[w] = k4 + 4 < nj[w] ? __ldg(src[w] + k4 + 4) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int w = 0; w < kCheckRows; w++) {
          const int j = j0 + 8 * w + (int)(lane >> 2);
          const int8_t* qj = qs + __shfl_sync(0xFFFFFFFFu, q, j) * ld;
          auto val = [&](uint32_t x) {
            const uint32_t o = x & 0xFFFFu;
            return ((int)x >> 16) * (a.sgn ? (int)qj[o] : (int)(uint8_t)qj[o]);
          };
          auto dot = [&](uint4 x) { return val(x.x) + val(x.y) + val(x.z) + val(x.w); };
          int x = dot(x0[w]) + dot(x1[w]);
          for (uint32_t k4 = (lane & 3u) + 8; k4 < nj[w]; k4 += 8) {
            const uint4 y0 = __ldg(src[w] + k4);
            const uint4 y1 = k4 + 4 < nj[w] ? __ldg(src[w] + k4 + 4) : make_uint4(0u, 0u, 0u, 0u);
            x += dot(y0) + dot(y1);
          }
          __syncwarp();
          x += __shfl_xor_sync(0xFFFFFFFFu, x, 1);
          x += __shfl_xor_sync(0xFFFFFFFFu, x, 2);
          // lane j0 + 8 w + g takes the sum of the four lanes 4 g .. 4 g + 3
          const int y = __shfl_sync(0xFFFFFFFFu, x, (int)(lane & 7u) * 4);
          if ((int)(lane >> 3) == j0 / 8 + w) score += y;
        }
      }
      const uint32_t key = a.rowscale && h < total
          ? key_f32(__fmul_rn(__int2float_rn(score), __ldg(a.rowscale + row))) : key_i32(score);
      if (h < total && key >= th) {
        const uint32_t o = atomicAdd(a.cnt + qp, 1u);
        if (o < a.cap) a.surv[qp * a.cap + o] = make_uint2(key, row);
      }
      __syncwarp();
    }
  }
}

}  // namespace dev
}  // namespace aes
