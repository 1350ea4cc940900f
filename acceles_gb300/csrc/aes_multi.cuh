// aes_multi.cuh -- candidate pass of a few queries: one read of the Ultra-CSR matrix scores four.
//
// The plain pass (aes_kernels.cuh) decodes every packet once per query and uses one byte of each
// 32-bit word it gathers from its lane-replicated query table.  Here the word of a column holds
// the bytes of four queries, so the flags, column windows, addresses and gathers of a packet serve
// four; what is added per group of four entries is the 4x4 byte transpose (8 PRMT) and three more
// dp4a, and per row the sums and compares of the other three queries.  Rows, packets, ranges and
// the carry between lanes are those of the plain pass.  Bound by instruction issue, as that pass
// is at 6 and 4 bits: four queries take about 1.9 times the time of one (whole calls, four queries
// of a 4M x 1024 8-bit matrix 185 -> 114 us, of 1M x 1024 6-bit with 32 partitions 127 -> 81 us).
// 24 warps per CTA: the state of four queries takes 80 registers, over the 64 of 32 warps.
#pragma once

#include "aes_batch.cuh"

namespace aes {
namespace dev {

constexpr int kMultiQ = 4;       // queries per matrix read
constexpr int kMultiWarps = 24;
constexpr int kMultiThreads = kMultiWarps * 32;

struct MultiArgs {
  const uint4* tiles;
  const uint32_t* tile_rowbase;
  uint32_t n_tiles, n_rows, cols;
  const int8_t* q8;             // [nq][q8_ld]
  uint32_t q8_ld, nq;           // blockIdx.y scores queries 4 y .. 4 y + 3
  const float* rowscale;
  uint32_t split, slice;
  const uint32_t* thr;          // [nq][split]
  uint32_t* cnt;                // [nq][split]
  uint2* surv;                  // [nq][split][cap]
  uint32_t cap;
  uint32_t* keys_out;           // sample pass: [nq][keys_ld]
  uint32_t keys_ld;
  const uint32_t* sample_first; // owned-row offset per sample tile
  uint32_t sample_stride, n_sample_tiles;
};

__host__ inline size_t multi_smem_bytes(uint32_t cols, uint32_t split) {
  return (size_t)cols * kPlainTableBytesPerCol + (size_t)kMultiWarps * kPlainTileBuf +
         (split <= kThrSmemMax ? (size_t)split * kMultiQ * 4 : 0);
}

// Thresholds and survivors of the CTA's four queries.  A row is compared with bounds on what the
// pass computes, the packet sums (integer keys; signed 6-bit sums are four times the score) or
// rowscale * score as FP32 (SCALED); past a bound it is checked against its own partition's key.
template <int SHIFT, bool SCALED>
struct MultiEmit {
  const MultiArgs& a;
  const uint32_t* thr_s;  // [split][4] in shared memory, or nullptr
  uint32_t q0, nq;        // first query, queries (1 .. 4)
  __device__ __forceinline__ uint32_t thr_key(uint32_t p, int t) const {
    if (thr_s) return thr_s[p * kMultiQ + t];
    return (uint32_t)t < nq ? a.thr[(size_t)(q0 + t) * a.split + p] : 0xFFFFFFFFu;
  }
  // the bound of a key threshold: x >= bound (signed, or FP32 bits) <=> key(x) >= th
  __device__ __forceinline__ static int32_t bound(uint32_t th) {
    if constexpr (SCALED) {  // x >= +0: key(x) = bits(x) | 2^31, and bits of x >= 0 order as integers
      return th <= 0x80000000u ? 0 : (int32_t)(th & 0x7FFFFFFFu);
    } else {
      const int32_t b = (int32_t)(th ^ 0x80000000u);
      constexpr int32_t lim = 0x7FFFFFFF >> SHIFT;
      return b > lim ? 0x7FFFFFFF : (b < -lim ? (int32_t)0x80000000u : b * (1 << SHIFT));
    }
  }
  // per query, the lowest bound over the partitions of rows r0 .. r1
  __device__ __forceinline__ void bounds(uint32_t r0, uint32_t r1, int32_t (&b)[kMultiQ]) const {
    const uint32_t p0 = part_of(r0, a.split, a.slice), p1 = part_of(r1, a.split, a.slice);
#pragma unroll
    for (int t = 0; t < kMultiQ; t++) b[t] = bound(thr_key(p0, t));
    for (uint32_t p = p0 + 1; p <= p1; p++)
#pragma unroll
      for (int t = 0; t < kMultiQ; t++) b[t] = min(b[t], bound(thr_key(p, t)));
  }
  __device__ __forceinline__ void operator()(bool valid, uint32_t row, const uint32_t (&sum)[kMultiQ],
                                             const int32_t (&b)[kMultiQ]) const {
    int32_t x[kMultiQ];
    if constexpr (SCALED) {
      const float rs = valid ? __ldg(a.rowscale + row) : 0.0f;
#pragma unroll
      for (int t = 0; t < kMultiQ; t++)
        x[t] = (int32_t)__float_as_uint(__fmul_rn(__int2float_rn((int32_t)sum[t]), rs));
    } else {
#pragma unroll
      for (int t = 0; t < kMultiQ; t++) x[t] = (int32_t)sum[t];
    }
    const bool hit = (x[0] >= b[0]) | (x[1] >= b[1]) | (x[2] >= b[2]) | (x[3] >= b[3]);
    if (valid && hit) {
      const uint32_t p = part_of(row, a.split, a.slice);
#pragma unroll
      for (int t = 0; t < kMultiQ; t++) {
        const uint32_t key = SCALED ? key_f32(__uint_as_float((uint32_t)x[t])) : key_i32(x[t] >> SHIFT);
        if (key >= thr_key(p, t) && (uint32_t)t < nq) {
          const size_t qp = (size_t)(q0 + t) * a.split + p;
          const uint32_t i = atomicAdd(a.cnt + qp, 1u);
          if (i < a.cap) a.surv[qp * a.cap + i] = make_uint2(key, row);
        }
      }
    }
  }
};

// The sample pass: every row's key, query-major
template <int SHIFT, bool SCALED>
struct MultiSampleEmit {
  const MultiArgs& a;
  uint32_t q0, nq;
  uint32_t base;  // first owned row of the tile minus its key index
  __device__ __forceinline__ void bounds(uint32_t, uint32_t, int32_t (&b)[kMultiQ]) const {
#pragma unroll
    for (int t = 0; t < kMultiQ; t++) b[t] = 0;
  }
  __device__ __forceinline__ void operator()(bool valid, uint32_t row, const uint32_t (&sum)[kMultiQ],
                                             const int32_t (&)[kMultiQ]) const {
    if (!valid) return;
    const float rs = SCALED ? __ldg(a.rowscale + row) : 0.0f;
#pragma unroll
    for (int t = 0; t < kMultiQ; t++) {
      const int32_t sc = (int32_t)sum[t] >> SHIFT;
      const uint32_t key = SCALED ? key_f32(__fmul_rn(__int2float_rn(sc), rs)) : key_i32(sc);
      if ((uint32_t)t < nq) a.keys_out[(size_t)(q0 + t) * a.keys_ld + (row - base)] = key;
    }
  }
};

// Running sums of one lane's packet (Rows8 of the plain pass, for four queries)
struct Rows4x {
  int32_t S[kMultiQ];
  uint32_t first[kMultiQ], prev[kMultiQ];
  uint32_t row;
  bool seen;
};

template <int B, bool SGN>
struct MultiSpans {
  using D = PacketSpans<B, SGN>;
  using Flags = typename D::Flags;
  static constexpr int P = D::P, NG = D::NG;

  // the four values of group G, and per query the four bytes at its columns
  template <int G>
  __device__ __forceinline__ static void load_group(const uint32_t (&w)[16], const char* qtb,
                                                    uint32_t lane4, uint32_t (&V)[kMultiQ], uint32_t& v4) {
    constexpr int J = 4 * G;
    constexpr int n = (P - J) < 4 ? (P - J) : 4;
    uint32_t W[4] = {0u, 0u, 0u, 0u};
    W[0] = D::template qval<J>(w, qtb, lane4);
    if constexpr (n > 1) W[1] = D::template qval<(n > 1 ? J + 1 : J)>(w, qtb, lane4);
    if constexpr (n > 2) W[2] = D::template qval<(n > 2 ? J + 2 : J)>(w, qtb, lane4);
    if constexpr (n > 3) W[3] = D::template qval<(n > 3 ? J + 3 : J)>(w, qtb, lane4);
    transpose4(W, V);
    v4 = D::unpack(D::template field32<11 * P + B * J>(w));
    if constexpr (n < 4) v4 &= (1u << (8 * n)) - 1u;
  }

  // running sums at flag j of a span of NGR groups
  template <int NGR>
  __device__ __forceinline__ static void prefix(int j, const int32_t (&Sa)[kMultiQ],
                                                const uint32_t (&V)[3][kMultiQ], const uint32_t (&v)[3],
                                                uint32_t (&out)[kMultiQ]) {
    const uint64_t m = ~(~0ull << (8 * (j & 7)));  // bytes before entry j (j < 8)
    uint32_t ma = v[0] & (uint32_t)m, mb = v[1] & (uint32_t)(m >> 32), mc = 0u;
    if constexpr (NGR == 3) {
      const bool lo = j < 8;
      ma = lo ? ma : v[0];
      mb = lo ? mb : v[1];
      mc = lo ? 0u : v[2] & ~(0xFFFFFFFFu << (8 * ((j - 8) & 3)));
    }
#pragma unroll
    for (int t = 0; t < kMultiQ; t++) {
      int32_t x = D::dot4(mb, V[1][t], D::dot4(ma, V[0][t], Sa[t]));
      if constexpr (NGR == 3) x = D::dot4(mc, V[2][t], x);
      out[t] = (uint32_t)x;
    }
  }

  template <int G, bool INNER, class OnRow>
  __device__ __forceinline__ static void span(const uint32_t (&w)[16], const char* qtb,
                                              uint32_t lane4, Flags F, bool multi, Rows4x& s,
                                              const OnRow& on_row) {
    if constexpr (G < NG) {
      constexpr int NGR = D::template span_groups<G>();
      uint32_t V[3][kMultiQ], v[3] = {0u, 0u, 0u};
      load_group<G>(w, qtb, lane4, V[0], v[0]);
      load_group<G + 1>(w, qtb, lane4, V[1], v[1]);
      if constexpr (NGR == 3) load_group<(NGR == 3 ? G + 2 : G)>(w, qtb, lane4, V[2], v[2]);
      int32_t Sa[kMultiQ];
#pragma unroll
      for (int t = 0; t < kMultiQ; t++) {
        Sa[t] = s.S[t];
        s.S[t] = D::dot4(v[1], V[1][t], D::dot4(v[0], V[0][t], Sa[t]));
        if constexpr (NGR == 3) s.S[t] = D::dot4(v[2], V[2][t], s.S[t]);
      }
      const uint32_t fP = (uint32_t)((F & (Flags)D::template span_bits<G>()) >> (4 * G));
      const bool has = fP != 0;
      uint32_t at[kMultiQ];
      prefix<NGR>(__ffs(fP) - 1, Sa, V, v, at);
      if constexpr (INNER) {
        uint32_t sc[kMultiQ];
#pragma unroll
        for (int t = 0; t < kMultiQ; t++) sc[t] = at[t] - s.prev[t];
        on_row(has && s.seen, s.row, sc);
      }
#pragma unroll
      for (int t = 0; t < kMultiQ; t++) {
        s.first[t] = (has && !s.seen) ? at[t] : s.first[t];
        s.prev[t] = has ? at[t] : s.prev[t];
      }
      s.row += has ? 1u : 0u;
      s.seen = s.seen || has;
      if (multi) {
        uint32_t rest = fP & (fP - 1u);
        while (rest) {
          const int j = __ffs(rest) - 1;
          rest &= rest - 1u;
          prefix<NGR>(j, Sa, V, v, at);
          if constexpr (INNER) {
            uint32_t sc[kMultiQ];
#pragma unroll
            for (int t = 0; t < kMultiQ; t++) sc[t] = at[t] - s.prev[t];
            on_row(true, s.row, sc);
          }
#pragma unroll
          for (int t = 0; t < kMultiQ; t++) s.prev[t] = at[t];
          s.row++;
        }
      }
      span<G + NGR, INNER>(w, qtb, lane4, F, multi, s, on_row);
    }
  }
};

struct MultiState {
  bool open_owned;
  uint32_t startG[kMultiQ], carryG[kMultiQ];
};
struct MultiPart {  // partition of the tile's first row, followed across tiles
  uint32_t end;     // first row past it (0xFFFFFFFF: it is the last)
  int32_t b[kMultiQ];
};

// One tile of a warp's range; true once the range is complete (tile_step of the plain pass)
template <int B, bool SGN, bool SCALED, bool CLOSING, class Emit>
__device__ __forceinline__ bool multi_step(const MultiArgs& a, uint32_t t, const uint32_t (&w)[16],
                                           uint32_t rowbase, MultiState& st, const Emit& emit,
                                           const char* qtb, MultiPart& pt) {
  using D = PacketSpans<B, SGN>;
  using Flags = typename D::Flags;
  const uint32_t lane = threadIdx.x & 31u;
  if constexpr (CLOSING) {
    if (t >= a.n_tiles) {  // the end of the matrix closes the last row
      int32_t b[kMultiQ];
      uint32_t sc[kMultiQ];
      emit.bounds(a.n_rows - 1, a.n_rows - 1, b);
#pragma unroll
      for (int q = 0; q < kMultiQ; q++) sc[q] = st.carryG[q] - st.startG[q];
      emit(st.open_owned && lane == 0, a.n_rows - 1, sc, b);
      return true;
    }
  }
  const Flags F = PacketDecoder<B, SGN>::flags(w);
  const uint32_t has_mask = __ballot_sync(0xFFFFFFFFu, F != 0);
  uint32_t rbase = rowbase;
  int32_t b[kMultiQ];
  if constexpr (!CLOSING) {
    const uint32_t nf = popc_flags(F);
    const uint32_t incl = warp_incl_sum(nf, lane);
    rbase += incl - nf;
    const uint32_t r1 = rowbase + __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (rowbase >= pt.end) {  // the tile starts in a later partition
      const uint32_t p = part_of(rowbase, a.split, a.slice);
      pt.end = (p + 1 >= a.split) ? 0xFFFFFFFFu : (p + 1) * a.slice;
      emit.bounds(rowbase, rowbase, pt.b);
    }
    if (r1 < pt.end) {
#pragma unroll
      for (int q = 0; q < kMultiQ; q++) b[q] = pt.b[q];
    } else {
      emit.bounds(rowbase, r1, b);
    }
  }
  auto on_row = [&](bool valid, uint32_t row, const uint32_t (&sc)[kMultiQ]) { emit(valid, row, sc, b); };
  const bool multi = !CLOSING && __any_sync(0xFFFFFFFFu, D::two_in_a_span(F));
  Rows4x s{{0, 0, 0, 0}, {0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}, rbase, false};
  MultiSpans<B, SGN>::template span<0, !CLOSING>(w, qtb, lane << 2, F, multi, s, on_row);
  uint32_t LB[kMultiQ], sum[kMultiQ];
#pragma unroll
  for (int q = 0; q < kMultiQ; q++) {
    const uint32_t total = (uint32_t)s.S[q];
    const uint32_t incl = warp_incl_sum(total, lane);
    LB[q] = st.carryG[q] + incl - total;
    sum[q] = __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  if constexpr (CLOSING) {
    if (has_mask == 0) {
#pragma unroll
      for (int q = 0; q < kMultiQ; q++) st.carryG[q] += sum[q];
      return false;
    }
    uint32_t sc[kMultiQ];
#pragma unroll
    for (int q = 0; q < kMultiQ; q++) sc[q] = LB[q] + s.first[q] - st.startG[q];
    emit.bounds(rowbase, rowbase, b);
    emit(lane == (uint32_t)(__ffs(has_mask) - 1) && st.open_owned, rowbase, sc, b);
    return true;
  } else {
    const uint32_t left = has_mask & ((1u << lane) - 1u);
    const uint32_t from = left ? (31 - __clz(left)) : 0u;
    uint32_t sc[kMultiQ];
#pragma unroll
    for (int q = 0; q < kMultiQ; q++) {
      const uint32_t lastGb = LB[q] + s.prev[q];
      const uint32_t inh = __shfl_sync(0xFFFFFFFFu, lastGb, from);
      sc[q] = LB[q] + s.first[q] - (left ? inh : st.startG[q]);
      if (has_mask) st.startG[q] = __shfl_sync(0xFFFFFFFFu, lastGb, 31 - __clz(has_mask));
      st.carryG[q] += sum[q];
    }
    on_row(F && (left || st.open_owned), rbase, sc);
    if (has_mask) st.open_owned = true;
    return false;
  }
}

// One warp streams tiles [tb, te) (cand_range of the plain pass)
template <int B, bool SGN, bool SCALED, class Emit>
__device__ void multi_range(const MultiArgs& a, uint32_t tb, uint32_t te, const Emit& emit,
                            const char* qtb, uint4* stg) {
  const uint32_t lane = threadIdx.x & 31u;
  if (tb >= te) return;
  MultiState st{tb == 0, {0u, 0u, 0u, 0u}, {0u, 0u, 0u, 0u}};
  MultiPart pt;
  {
    const uint32_t r0 = __ldg(a.tile_rowbase + tb);
    const uint32_t p = part_of(r0, a.split, a.slice);
    pt.end = (p + 1 >= a.split || a.slice == 0) ? 0xFFFFFFFFu : (p + 1) * a.slice;
    emit.bounds(r0, r0, pt.b);
  }
  uint32_t w[16];
  uint32_t rn = 0;
  auto fetch = [&](uint32_t t) {
    if (t < a.n_tiles) {
      const uint4* src = a.tiles + (size_t)t * 128 + lane;
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stg + s * 32 + lane);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + s * 32)
                     : "memory");
      }
      rn = __ldg(a.tile_rowbase + t);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  fetch(tb);
  for (uint32_t t = tb;; t++) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const uint4 v = stg[s * 32 + lane];
      w[4 * s + 0] = v.x;
      w[4 * s + 1] = v.y;
      w[4 * s + 2] = v.z;
      w[4 * s + 3] = v.w;
    }
    const uint32_t r = rn;
    if (t + 1 <= te) fetch(t + 1);
    if (t < te) {
      multi_step<B, SGN, SCALED, false>(a, t, w, r, st, emit, qtb, pt);
    } else if (multi_step<B, SGN, SCALED, true>(a, t, w, r, st, emit, qtb, pt)) {
      return;
    }
    if (t + 1 > te) fetch(t + 1);
  }
}

template <int B, bool SGN, bool SCALED, bool SAMPLE>
__global__ void __launch_bounds__(kMultiThreads, 1) k_cand_multi(MultiArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);
  const char* qtb = reinterpret_cast<const char*>(smem);  // qt[cols][32 lanes]
  unsigned char* after = smem + (size_t)a.cols * kPlainTableBytesPerCol;
  uint4* stg = reinterpret_cast<uint4*>(after) + (size_t)warp * (kPlainTileBuf / 16);
  uint32_t* thr_s = reinterpret_cast<uint32_t*>(after + kMultiWarps * kPlainTileBuf);
  const uint32_t q0 = blockIdx.y * kMultiQ, nq = min((uint32_t)kMultiQ, a.nq - q0);
  if constexpr (SAMPLE) {  // (the filter's queries were quantised before the sample pass)
    grid_wait();
    grid_next();
  }
  {  // the columns' words through the tile buffers' area (4 KB), then one copy per lane
    uint32_t* qstage = reinterpret_cast<uint32_t*>(after);
    const int8_t* q8 = a.q8 + (size_t)q0 * a.q8_ld;
    for (uint32_t c = threadIdx.x; c < a.cols; c += kMultiThreads) {
      uint32_t v = 0;
#pragma unroll
      for (uint32_t t = 0; t < kMultiQ; t++)
        v |= t < nq ? (uint32_t)(uint8_t)q8[(size_t)t * a.q8_ld + c] << (8 * t) : 0u;
      qstage[c] = v;
    }
    __syncthreads();
    uint4* qt = reinterpret_cast<uint4*>(smem);
    for (uint32_t i = threadIdx.x; i < a.cols * 8u; i += kMultiThreads) {
      const uint32_t v = qstage[i >> 3];
      qt[i] = make_uint4(v, v, v, v);
    }
  }
  const uint32_t gw = blockIdx.x * kMultiWarps + warp, nw = gridDim.x * kMultiWarps;
  constexpr int SHIFT = SCALED ? 0 : PacketSpans<B, SGN>::kScoreShift;
  if constexpr (SAMPLE) {
    __syncthreads();
    for (uint32_t i = gw; i < a.n_sample_tiles; i += nw) {
      const uint32_t t = i * a.sample_stride;
      const MultiSampleEmit<SHIFT, SCALED> em{a, q0, nq, __ldg(a.sample_first + i)};
      multi_range<B, SGN, SCALED>(a, t, t + 1, em, qtb, stg);
    }
    return;
  }
  grid_wait();
  // (one partition too: 40 queries of 2M x 1024, 8 bits, the whole call 324 us; with its four thresholds
  // read from global memory between a hit's atomics 340, before them 335 and 24 bytes of spills)
  const bool in_smem = a.split <= kThrSmemMax;
  if (in_smem)
    for (uint32_t i = threadIdx.x; i < a.split * kMultiQ; i += kMultiThreads) {
      const uint32_t p = i / kMultiQ, t = i % kMultiQ;
      thr_s[i] = t < nq ? a.thr[(size_t)(q0 + t) * a.split + p] : 0xFFFFFFFFu;
    }
  __syncthreads();
  const uint64_t n = a.n_tiles;
  const uint32_t tb = (uint32_t)((n * gw) / nw), te = (uint32_t)((n * (gw + 1)) / nw);
  const MultiEmit<SHIFT, SCALED> em{a, in_smem ? thr_s : nullptr, q0, nq};
  multi_range<B, SGN, SCALED>(a, tb, te, em, qtb, stg);
}

}  // namespace dev
}  // namespace aes
