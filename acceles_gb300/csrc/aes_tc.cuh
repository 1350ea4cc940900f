// aes_tc.cuh -- candidate pass on the tensor cores (tcgen05): exact for 4-bit matrices, and the kernel of
// the filter for the other widths (aes_tf.cuh).
//
// The batched candidate pass of aes_batch.cuh scores 128 queries per matrix read with dp4a and is
// bound by instruction issue.  For B = 4 every matrix value (signed [-8, 7], unsigned [0, 15]) and
// every quantised query value is an integer of magnitude <= 16, which FP8 e4m3 holds exactly, and
// every partial sum of a row score stays far below 2^24 (15 * 15 * 1024), so an FP32 accumulation
// of the products is exact in any order.  The pass is then a dense product
//
//     D[128 rows x 128 queries] = A[128 rows x cols] * Q[128 queries x cols]^T
//
// per tile of 128 consecutive rows, with the row tile A densified in shared memory:
//   - the host lays out the quantised entries per (row tile, 256-column chunk) as 32-bit words
//     holding the entry's byte offset inside the chunk's operand layout and its e4m3 byte;
//   - producer warps write a chunk's entries into one of two or three zeroed 32 KB chunk buffers
//     (and write them back to zero once the MMAs of that chunk have read the buffer);
//   - the MMA warp's elected thread issues the chunk's tcgen05.mma (kind::f8f6f4, M = 128, N = 128,
//     K = 32 each) into one of four 128-column FP32 accumulators in tensor memory; tcgen05.commit
//     signals mbarriers when a chunk buffer is read and when a tile's accumulator is complete;
//   - epilogue warps read a complete accumulator with tcgen05.ld while the next tiles' MMAs run and
//     compare every (row, query) score with the query's threshold; a hit goes into the CTA's queue
//     (device memory, in practice L2), a filter's into its lists for k_recheck;
//   - two warps drain the queues, appending the hits to the queries' survivors as the same
//     candidate keys as in the other passes, so that no epilogue warp waits on an atomic's round trip.
// Two blocks of 128 queries run together on CTA pairs (cta_group::2, M = 256 over the pair's two
// row tiles, N = 256 queries): the same roles in each CTA, the even CTA's thread issuing the MMAs
// (see k_cand_tc).
// The roles hand work over through mbarriers only.
// Both operands are K-major without swizzle (layout in aes_tc_layout.h).
// Reference counterpart: the candidate pass spmv_ucsr_top_k_multicore.hpp:195-413 (one query per
// pass on the FPGA); scores equal those of gold_algorithms.hpp:249-308 on the same integers.
#pragma once

#include "aes_kernels.cuh"
#include "aes_tc_layout.h"

namespace aes {
namespace dev {

// Warp roles: warps 0-8 stage the chunks (producers, a group of three or four warps per chunk
// buffer), one thread of warp 9 issues the MMAs (on a pair: the even CTA's; the warp also allocates
// tensor memory), warps 10 and 11 append the hits, the warps from 12 on read the accumulators (warp w
// may only read tensor-memory lanes 32 (w % 4) .. + 31; each four warps take a share of the queries).
// They hand work over through mbarriers only.
constexpr int kTcMmaWarp = 9;
constexpr int kTcDrainWarp = 10;  // and the one after it: unit t's hits are appended by 10 + t % 2
constexpr uint32_t kTcDrains = 2;
constexpr int kTcEpiWarp = 12;
// producers of a chunk buffer, with nb buffers
__host__ __device__ constexpr uint32_t tc_group(uint32_t nb) { return nb == 3 ? 96u : 128u; }
constexpr uint32_t kTcTmemCols = 512;  // all of tensor memory, in FP32 accumulators
// Queries per launch and accumulators.  One CTA: 128 queries (N = 128, M = 128), four
// accumulators of 128 columns.  A CTA pair (cta_group::2): 256 queries (N = 256, each CTA
// holding 128 of them in its operand) and M = 256 (each CTA's 128-row tile), two accumulators
// of 256 columns in each CTA's tensor memory.
template <bool PAIR>
struct TcShape {
  static constexpr uint32_t Q = PAIR ? 2 * kTcQ : kTcQ;
  static constexpr uint32_t ACC = kTcTmemCols / Q;
  // epilogue threads, 32 or 64 queries each: a warp's reads of an accumulator are a chain of
  // latencies, and a pair's two accumulators leave little time for it (2M rows x 1024, 64M entries,
  // 256 queries: 286 us with 8 warps, 278 with 16; 128 queries on one CTA: 203 and 215)
  static constexpr uint32_t EPI = PAIR ? 512 : 256;
  static constexpr uint32_t THREADS = kTcEpiWarp * 32 + EPI;
};
// mbarriers of a kernel with nb chunk buffers and acc accumulators: staged[nb] (producers ->
// MMA), done[nb] (MMA -> producers), full[acc] (MMA -> epilogue), empty[acc] (epilogue -> MMA),
// drain (the MMA thread's own MMAs complete), queued[kTcQueues] (epilogue -> drain warp),
// drained[kTcQueues] (drain warp -> epilogue); then the tensor-memory address, the give-up flag
// and the counts of the hit queues
constexpr uint32_t kTcQueues = 6;       // units whose hits may wait (a long row hits for most queries)
constexpr uint32_t kTcLists = 2 * kTcQ / 32;
static_assert(kTcLists >= kTcQueues, "counts of queues and lists share their place");
__host__ __device__ constexpr uint32_t tc_nbars(uint32_t nb, uint32_t acc) {
  return 2 * nb + 2 * acc + 1 + 2 * kTcQueues;
}
constexpr uint32_t kTcQueueMax = 4096;  // hits of a unit that its queue holds at most

// shared memory of one CTA of the pass with nb chunk buffers (2 or 3)
__host__ inline size_t tc_smem_bytes(uint32_t cols, uint32_t split, uint32_t nb, bool pair) {
  const uint32_t S = split <= 1 ? 1 : split;
  const uint32_t q = pair ? 2 * kTcQ : kTcQ;
  return tc_qtab_bytes(cols) + nb * (size_t)kTcChunkBytes + (size_t)S * q * 4 +
         ((tc_nbars(nb, kTcTmemCols / q) * 8 + 8 + kTcLists * 4 + 15) & ~15u);
}
// chunk buffers for a configuration: three where they fit next to the query operand and the
// thresholds (the producers then run two chunks ahead of the MMAs), else two
__host__ inline uint32_t tc_bufs(uint32_t cols, uint32_t split, size_t smem_limit, bool pair) {
  return tc_smem_bytes(cols, split, 3, pair) <= smem_limit ? 3u : 2u;
}

// e4m3 query operand of queries q0 .. q0 + nq - 1 (zero past nq and past cols)
__global__ void k_qtable_tc(const int8_t* q8, uint32_t ld8, uint32_t cols, uint32_t q0,
                            uint32_t nq, uint8_t* __restrict__ qt) {
  grid_wait();
  grid_next();
  const uint32_t kp = tc_kpad(cols);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kTcQ * kp) return;
  const uint32_t n = i / kp, k = i % kp;
  const int v = (n < nq && k < cols) ? (int)q8[(size_t)(q0 + n) * ld8 + k] : 0;
  qt[tc_off(n, k)] = e4m3_small(v);
}

struct TcArgs {
  const uint32_t* ent;   // per entry: byte offset in its chunk operand << 16 | e4m3 value
  const uint32_t* ptr;   // [n_rtiles * nch + 1] first entry of (row tile, chunk)
  uint32_t n_rtiles, nch, kpad, n_rows;
  const uint8_t* qt;     // e4m3 query operand of this launch, tc_qtab_bytes(cols)
  uint32_t q0, nq;       // this launch scores queries q0 .. q0 + nq - 1 (nq <= 128, on pairs 256)
  const float* rowscale;
  // filter of approximate scores (aes_tf.cuh), or null: per row {sum |v'| << 13 | ceil(sum |d| / 2),
  // sum v}, and the launch's query statistics
  const uint2* rowstat;
  const uint32_t* qstat;
  uint32_t split, slice; // split >= 1
  const uint32_t* thr;   // [nq_total][split]
  uint32_t* cnt;         // [nq_total][split]
  uint2* surv;           // [nq_total][split][cap]
  uint32_t cap;
  uint32_t* status;      // [nq_total]
  // [gridDim.x][kTcQueues][queue_cap] hit queues of successive units; a filter's lists of the rows it
  // lets through, [gridDim.x][kTcLists][queue_cap] {row, mask of queries} per block of 32 queries,
  // and their counts
  uint2* queue;
  uint32_t* list_n;      // [gridDim.x][kTcLists]
  uint32_t queue_cap;
  uint32_t mma_idle;     // failure-path test: the MMA role issues nothing, so every hand-over
                         // wait of the other roles runs out and the CTA gives up
};

__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// shared-memory operand descriptor: start address, K-adjacent core matrices 2048 B apart
// (leading byte offset), 8-row groups 128 B apart (stride byte offset), descriptor version 1,
// no swizzle
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(2048u >> 4) << 16) |
         ((uint64_t)(128u >> 4) << 32) | ((uint64_t)1 << 46);
}
// Scope: what crosses the CTAs of a pair is waited for at cluster scope, relaxed, behind it a fence that
// acquires shared memory or the tcgen05 fence of the caller.
enum TcScope { TC_CTA, TC_CLUSTER, TC_CLUSTER_RELAXED };
template <TcScope SCOPE = TC_CTA>
__device__ __forceinline__ uint32_t tc_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if constexpr (SCOPE == TC_CTA)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  if constexpr (SCOPE == TC_CLUSTER)
    if (done) asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
  return done;
}
// Waits for the phase of the given parity to complete, for about a second at most, whether or
// not another role has given up: the MMA thread's wait for its own MMAs in flight before the CTA
// frees its tensor memory and leaves.
template <TcScope SCOPE = TC_CTA>
__device__ __forceinline__ bool tc_wait_own(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  uint32_t done = 0;
  while (!done) {
    done = tc_try<SCOPE>(bar, parity);
    if (!done && clock64() - t0 > (1ll << 31)) return false;
  }
  return true;
}
// Waits for the phase of the given parity to complete.  Gives up after about a second, or as
// soon as another thread of the CTA has given up (*gave_up set), so that every role leaves its
// loop instead of waiting on a partner that has left.
template <TcScope SCOPE = TC_CTA>
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up) {
  const long long t0 = clock64();
  uint32_t done = 0;
  while (!done) {
    done = tc_try<SCOPE>(bar, parity);
    if (done) break;
    if (*gave_up) return false;
    if (clock64() - t0 > (1ll << 31)) {
      *gave_up = 1u;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void tc_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// A warp's arrival, once for its 32 threads.  PAIR: on the barrier at the same offset in the pair's even
// CTA (the one whose thread issues the MMAs), through its shared::cluster address and at cluster scope,
// relaxed.  BYTES: operand bytes in shared memory are handed over, released by a fence for shared memory
// alone (a plain release also waits for global memory: 256 queries of 8M rows x 1024, 256M entries,
// 1080 us a launch where this takes 1042); else only tensor-memory reads, which tcgen05.fence has ordered.
// The odd CTA's producers arrive on their own CTA's barrier, and its MMA warp, which has no MMAs to
// issue, passes each phase on: the fence is off the producers' path (1046 us on it).
template <bool PAIR, bool BYTES>
__device__ __forceinline__ void tc_arrive_warp(uint32_t bar) {
  __syncwarp();
  if ((threadIdx.x & 31u) == 0) {
    if constexpr (PAIR) {
      uint32_t ra;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(ra) : "r"(bar));
      if constexpr (BYTES) asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
      asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" :: "r"(ra) : "memory");
    } else {
      tc_arrive(bar);
    }
  }
}
template <bool PAIR>
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc,
                                       uint32_t acc) {
  if constexpr (PAIR) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n"
        :: "r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc));
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n"
        :: "r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc));
  }
}
// one thread of the warp, the same each time
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}
// Arrives on `bar` once the MMAs issued so far complete.  PAIR: on the barrier at the same
// offset in each CTA of ctamask (bit r: the pair's CTA of rank r).
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint32_t bar, uint16_t ctamask = 3) {
  if constexpr (PAIR) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        :: "r"(bar), "h"(ctamask) : "memory");
  } else {
    (void)ctamask;
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(bar) : "memory");
  }
}
// Tensor memory of the CTA (PAIR: of both CTAs, the same columns, by one warp of each)
template <bool PAIR>
__device__ __forceinline__ void tc_alloc(uint32_t slot) {
  if constexpr (PAIR) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(slot), "n"(kTcTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(slot), "n"(kTcTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
}
template <bool PAIR>
__device__ __forceinline__ void tc_dealloc(uint32_t tmem) {
  if constexpr (PAIR)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(kTcTmemCols));
  else
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(kTcTmemCols));
}
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 consecutive accumulator columns of this warp's 32 lanes (one row per thread)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// N scores of a row (FP32 bits) for consecutive queries that passed the epilogue's bound where
// `hit` has a bit: appended to the query's survivors if they pass the threshold itself.  qp: query
// and partition of the first; rs: the row's scale, negative without row scales.  The loads and the
// atomics of all N are in flight together.
template <int N>
__device__ __forceinline__ void tc_append(const TcArgs& a, uint32_t S, size_t qp, uint32_t row,
                                          const uint32_t* score, uint32_t hit, float rs) {
  uint32_t key[N], th[N], ix[N];
#pragma unroll
  for (int j = 0; j < N; j++) th[j] = (hit >> j) & 1u ? a.thr[qp + (size_t)j * S] : 0xFFFFFFFFu;
#pragma unroll
  for (int j = 0; j < N; j++) {
    const float f = __uint_as_float(score[j]);
    key[j] = rs >= 0.0f ? key_f32(__fmul_rn(f, rs)) : key_i32(__float2int_rn(f));
    if (key[j] < th[j]) hit &= ~(1u << j);
  }
#pragma unroll
  for (int j = 0; j < N; j++)
    if ((hit >> j) & 1u) ix[j] = atomicAdd(a.cnt + qp + (size_t)j * S, 1u);
#pragma unroll
  for (int j = 0; j < N; j++)
    if (((hit >> j) & 1u) && ix[j] < a.cap)
      a.surv[(qp + (size_t)j * S) * a.cap + ix[j]] = make_uint2(key[j], row);
}
// The hit queue of a unit: entries (query | row in tile << 8, score as FP32 bits); hits past its end
// are appended by the epilogue thread itself, the slots it had taken marked.  A filter: the CTA's
// lists
constexpr uint32_t kTcNoHit = 0xFFFFFFFFu;
struct TcQueue {
  uint2* e;
  uint32_t* n;    // entries taken (may pass cap)
  uint32_t cap;
};
// The thread's row of tile T, and its row scale (loaded before the accumulator wait, so that the
// load's latency passes while the MMAs finish)
__device__ __forceinline__ uint32_t tc_epi_row(uint32_t T) {
  return T * kTcRows + ((threadIdx.x >> 5) & 3u) * 32u + (threadIdx.x & 31u);
}
__device__ __forceinline__ float4 tc_lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
// The row's scale and sums on their way to L1 while its unit before is read, at no register: loaded
// when they are needed, they held an epilogue warp for 1000 of a unit's 5500 cycles (4M rows x 1024 at
// 8 bits, 512 queries, the whole call: 1726 -> 1674 us).
__device__ __forceinline__ void tc_prefetch(const TcArgs& a, uint32_t row) {
  if (row >= a.n_rows) return;
  if (a.rowscale) asm volatile("prefetch.global.L1 [%0];" :: "l"(a.rowscale + row));
  if (a.rowstat) asm volatile("prefetch.global.L1 [%0];" :: "l"(a.rowstat + row));
}
// two FP32 fused multiply-adds per instruction
__device__ __forceinline__ void tc_fma2(float& x0, float& x1, float a0, float a1, float b, float c0,
                                        float c1) {
  asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %4};\n"
      " mov.b64 c, {%5, %6};\n fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}\n"
      : "=f"(x0), "=f"(x1) : "f"(a0), "f"(a1), "f"(b), "f"(c0), "f"(c1));
}
// x[j] = score j times rs minus its bound (nthf: negated bounds, the same for every lane: 16-byte
// broadcasts)
__device__ __forceinline__ void tc_margin8(float (&x)[8], const uint32_t* v, float rs, float4 t0,
                                           float4 t1) {
  tc_fma2(x[0], x[1], __uint_as_float(v[0]), __uint_as_float(v[1]), rs, t0.x, t0.y);
  tc_fma2(x[2], x[3], __uint_as_float(v[2]), __uint_as_float(v[3]), rs, t0.z, t0.w);
  tc_fma2(x[4], x[5], __uint_as_float(v[4]), __uint_as_float(v[5]), rs, t1.x, t1.y);
  tc_fma2(x[6], x[7], __uint_as_float(v[6]), __uint_as_float(v[7]), rs, t1.z, t1.w);
}
// Query statistics of a filter launch: the centre c of the values (aes_tf.cuh: 512 + max, 512 - min)
__device__ __forceinline__ int tc_centre(const uint32_t* st) {
  const int hi = (int)st[0] - 512, lo = 512 - (int)st[1];
  return max(hi, -lo) <= 16 ? 0 : (hi + lo) / 2;
}
// Filter of approximate scores: minus what rs times the score may exceed rs times the approximate
// one by, rounded away from zero: c sum v + E sum |v'| + Q sum |d|, and for the FP32 arithmetic
// (the accumulator's, this one's and the compare's) 2^-12 of Q sum |v'| + |c sum v|.
// The accumulator takes a K = 32 step at a time, at most 32 of them (1024 columns), and each may
// lose 2^-23 of it, which stays below P = sum |v' q'| <= (Q + E) sum |v'| <= 1.1 Q sum |v'|: 2^-18 P in
// all.  That counts on sums that keep 24 bits within a step too, which PTX leaves open; measured, all
// of 1.4M accumulators equalled the exact sum (1024 columns; operands of 256 x 128, random, of
// alternating sign, ones after products of 27000, up to 2^25; every sum below 2^24 is then exact).
// The multiply-add and the compare round the score's distance from the bound by 2^-24 of it.  So 2^-12
// leaves a factor above 50.
__device__ __forceinline__ float tc_limit(uint2 st, int centre, float E, float Q, float rs) {
  const float r1 = (float)(st.x >> 13), r2 = 2.0f * (float)(st.x & 0x1FFFu);
  const float c = __fmul_ru((float)centre, __int2float_ru((int)st.y));
  float b = __fadd_ru(__fmul_ru(E, r1), __fmul_ru(Q, r2));
  b = __fadd_ru(b, 0.000244140625f * (Q * r1 + fabsf(c)));
  return -__fmul_ru(__fadd_ru(b, c), rs);
}
// Epilogue warps: reads accumulator `dbuf` of row tile T (thread = row, a share of the queries) and
// queues every (row, query) score at or above the query's bound.  nthf holds the negated bounds on
// rs * score (rs is the row's scale, or 1 without row scales, where the score is an exact integer),
// so a score passes where fma(score, rs, -bound) >= lim (0, or what an approximate score of the row
// may fall short by).  A block of 16 queries costs a fused
// multiply-add per two scores and the maximum of each group of eight (three-operand maxima); only
// groups that reach 0 are looked at again, and take their queue slots with one atomic per block.  The accumulator goes back to the MMA role (an
// arrive on `empty`) as soon as the thread's last load from it has completed.
// The epilogue was the pass's longest stage: a block with a hit waited for the survivor counter's
// atomic in device memory (over 1500 cycles; hits come in bursts, a long row passing for most of the
// queries), and each score took three instructions.  With the queues and the fused compares
// 2M rows x 1024, 64M entries, 256 queries: 748 -> 395 us (278 with the steps since).
template <bool PAIR>
__device__ __forceinline__ void tc_epilogue(const TcArgs& a, uint32_t T, uint32_t tmem,
                                            uint32_t dbuf, const float* nthf_all, uint32_t S,
                                            float rs, float lim, uint32_t empty,
                                            const TcQueue& hq) {
  constexpr uint32_t Q = TcShape<PAIR>::Q, WARPS = TcShape<PAIR>::EPI / 128;
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t g = warp & 3u, h = (warp - kTcEpiWarp) >> 2;
  const uint32_t row = tc_epi_row(T);
  const bool valid = row < a.n_rows;
  const uint32_t p = valid ? part_of(row, S, a.slice) : 0u;
  const uint32_t thaddr = tc_smem_u32(nthf_all + p * Q);
  // this warp's columns: an even share of those that the launch's queries fill, in blocks of 16 (half of
  // all, with 48 queries one half of the warps did the work: 2M rows x 1024, the whole call 360 -> 317 us)
  const uint32_t part = (min(a.nq, Q) + 16u * WARPS - 1u) / (16u * WARPS) * 16u;
  const uint32_t end = h * part + part;
  uint32_t mask = 0;  // a filter: hits of the block of 32 queries
#pragma unroll 1
  for (uint32_t col0 = h * part; col0 < end; col0 += 16u) {
    uint32_t v[16];
    float4 nt[4];  // read before the accumulator: both latencies pass together
#pragma unroll
    for (int j = 0; j < 4; j++) nt[j] = tc_lds4(thaddr + (col0 + 4u * j) * 4u);
    __syncwarp();  // tcgen05.ld needs the warp together again after a block with hits
    tc_ld16(tmem + dbuf * Q + col0 + ((g * 32u) << 16), v);
    if (col0 + 16u == end) {  // the last load of this unit has completed
      tc_fence_before();
      tc_arrive_warp<PAIR, false>(empty);
    }
    float m[2];
#pragma unroll
    for (int j8 = 0; j8 < 2; j8++) {
      float x[8];
      tc_margin8(x, v + 8 * j8, rs, nt[2 * j8], nt[2 * j8 + 1]);
      const float m0 = fmaxf(fmaxf(x[0], x[1]), x[2]), m1 = fmaxf(fmaxf(x[3], x[4]), x[5]);
      m[j8] = fmaxf(fmaxf(m0, m1), fmaxf(x[6], x[7]));
    }
    if (fmaxf(m[0], m[1]) >= lim && valid && col0 < a.nq) {
      uint32_t hit = 0;
#pragma unroll
      for (int j8 = 0; j8 < 2; j8++) {
        if (m[j8] >= lim) {
          float x[8];
          tc_margin8(x, v + 8 * j8, rs, nt[2 * j8], nt[2 * j8 + 1]);
#pragma unroll
          for (int j = 0; j < 8; j++) hit |= (x[j] >= lim ? 1u : 0u) << (8 * j8 + j);
        }
      }
      if (a.rowstat) {
        mask |= hit << (col0 & 16u);
      } else {
        const uint32_t nh = __popc(hit);
        uint32_t i = atomicAdd(hq.n, nh);
        const uint32_t meta = col0 | (row % kTcRows) << 8;
        if (i + nh <= hq.cap) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if ((hit >> j) & 1u) hq.e[i++] = make_uint2(meta + j, v[j]);
        } else {
          for (; i < hq.cap; i++) hq.e[i] = make_uint2(kTcNoHit, 0u);
          const size_t qp = (size_t)(a.q0 + col0) * S + p;
#pragma unroll
          for (int j8 = 0; j8 < 2; j8++)
            if ((hit >> (8 * j8)) & 255u)
              tc_append<8>(a, S, qp + (size_t)(8 * j8) * S, row, v + 8 * j8, hit >> (8 * j8),
                           a.rowscale ? rs : -1.0f);
        }
      }
    }
    if (mask && ((col0 & 16u) || col0 + 16u == end)) {
      const uint32_t l = col0 / 32u, k = atomicAdd(hq.n + l, 1u);
      if (k < hq.cap) hq.e[(size_t)l * hq.cap + k] = make_uint2(row, mask);
      mask = 0;
    }
  }
}

constexpr int kTcPer = 12;  // entries of a chunk a producer thread holds (1536 per chunk with two buffers, 1152 with three)

// A producer's share of one chunk's entries, G threads to a chunk: v[u] = entry b + t + G u for
// t + G u < n
template <uint32_t G>
struct TcEnt {
  uint32_t v[kTcPer];
  uint32_t b = 0, n = 0;
  __device__ __forceinline__ void load(const uint32_t* ent, uint32_t b_, uint32_t n_, uint32_t t) {
    b = b_;
    n = n_;
#pragma unroll
    for (int u0 = 0; u0 < kTcPer; u0 += 4) {
      if (u0 * G >= n) break;  // the whole group's
#pragma unroll
      for (int u = u0; u < u0 + 4; u++) {
        const uint32_t i = t + (uint32_t)u * G;
        v[u] = i < n ? __ldg(ent + b + i) : 0u;
      }
    }
  }
  // writes the entries' e4m3 bytes (or zeros) into a chunk buffer
  __device__ __forceinline__ void stage(unsigned char* ab, const uint32_t* ent, uint32_t t,
                                        bool clear) const {
#pragma unroll
    for (int u0 = 0; u0 < kTcPer; u0 += 4) {
      if (u0 * G >= n) break;
#pragma unroll
      for (int u = u0; u < u0 + 4; u++)
        if (t + (uint32_t)u * G < n) ab[v[u] >> 16] = clear ? (uint8_t)0 : (uint8_t)v[u];
    }
    for (uint32_t i = t + kTcPer * G; i < n; i += G) {
      const uint32_t e = __ldg(ent + b + i);
      ab[e >> 16] = clear ? (uint8_t)0 : (uint8_t)e;
    }
  }
};

// OR of `fail` over the G threads of a producer group (named barrier 1 + grp)
template <uint32_t G>
__device__ __forceinline__ bool tc_group_any(uint32_t grp, bool fail) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred f, r;\n setp.ne.u32 f, %1, 0;\n bar.red.or.pred r, %3, %2, f;\n"
      " selp.u32 %0, 1, 0, r;\n}\n"
      : "=r"(r) : "r"((uint32_t)fail), "n"(G), "r"(1u + grp) : "memory");
  return r != 0;
}


// A drain warp: appends n queued scores of row tile T, four per lane in flight
__device__ __forceinline__ void tc_drain_scores(const TcArgs& a, uint32_t S, const volatile uint2* hq,
                                                uint32_t n, uint32_t T) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t i0 = 0; i0 < n; i0 += 128u) {
    uint32_t meta[4], score[4], key[4], th[4], ix[4];
    size_t qp[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t i = i0 + u * 32u + lane;
      meta[u] = i < n ? hq[i].x : kTcNoHit;
      score[u] = i < n ? hq[i].y : 0u;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      th[u] = 0xFFFFFFFFu;
      key[u] = 0u;
      if (meta[u] != kTcNoHit) {
        const uint32_t row = T * kTcRows + (meta[u] >> 8);
        qp[u] = (size_t)(a.q0 + (meta[u] & 255u)) * S + part_of(row, S, a.slice);
        th[u] = a.thr[qp[u]];
        const float f = __uint_as_float(score[u]);
        key[u] = a.rowscale ? key_f32(__fmul_rn(f, __ldg(a.rowscale + row))) : key_i32(__float2int_rn(f));
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (meta[u] != kTcNoHit && key[u] >= th[u]) ix[u] = atomicAdd(a.cnt + qp[u], 1u);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (meta[u] != kTcNoHit && key[u] >= th[u] && ix[u] < a.cap)
        a.surv[qp[u] * a.cap + ix[u]] = make_uint2(key[u], T * kTcRows + (meta[u] >> 8));
  }
}
// One CTA per SM (PAIR: one CTA pair, a cluster of two, per two SMs), persistent over units of
// work U: a 128-row tile (one CTA), or two consecutive tiles, 2U for
// the even CTA and 2U + 1 for the odd one (PAIR).  Chunk i of the CTA is chunk i % nch of its
// unit i / nch; chunk buffer i % NB; accumulator (unit t) t % ACC.
// PAIR: the even CTA's MMA thread issues cta_group::2 MMAs with M = 256 (the two CTAs' row tiles
// from their own chunk buffers) and N = 256 (the two CTAs' 128-query operands), and commits them
// to the barriers of both CTAs; both CTAs' epilogues hand their accumulators back to the even CTA's
// barriers, and the odd CTA's staged chunks are passed on to them.  The two CTAs keep identical shared-memory
// layouts, since an operand descriptor addresses the same offset in both.
template <uint32_t NB, bool PAIR>
__global__ void __launch_bounds__(TcShape<PAIR>::THREADS, 1) k_cand_tc(TcArgs a) {
  grid_wait();
  static_assert(NB == 2 || NB == 3, "two or three chunk buffers");
  constexpr uint32_t Q = TcShape<PAIR>::Q, ACC = TcShape<PAIR>::ACC;
  constexpr uint32_t kDone = NB, kFull = 2 * NB, kEmpty = 2 * NB + ACC;
  constexpr uint32_t kDrain = kEmpty + ACC, kQueued = kDrain + 1, kDrained = kQueued + kTcQueues;
  constexpr uint32_t kBars = tc_nbars(NB, ACC);
  constexpr uint32_t G = tc_group(NB);  // producers of a chunk buffer
  // what crosses the pair is waited for at cluster scope (tc_arrive_warp)
  constexpr TcScope kAcq = PAIR ? TC_CLUSTER : TC_CTA, kRlx = PAIR ? TC_CLUSTER_RELAXED : TC_CTA;
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t qbytes = (a.kpad / 16u) * 2048u;
  unsigned char* sq = smem;                     // query operand (PAIR: this CTA's 128 queries)
  unsigned char* sa = smem + qbytes;            // NB chunk buffers of the row tile
  float* thf = reinterpret_cast<float*>(sa + NB * kTcChunkBytes);
  const uint32_t S = a.split <= 1 ? 1u : a.split;
  uint64_t* bars = reinterpret_cast<uint64_t*>(thf + S * Q);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + kBars);
  volatile uint32_t* gave_up = tslot + 1;
  uint32_t* hq_n = tslot + 2;  // [kTcLists]
  uint2* hq_e = a.queue + (size_t)blockIdx.x * (a.rowstat ? kTcLists : kTcQueues) * a.queue_cap;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  uint32_t rank = 0;  // the CTA's rank in its pair
  if constexpr (PAIR) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const uint32_t n_units = PAIR ? (a.n_rtiles + 1u) / 2u : a.n_rtiles;
  // units unit, unit + 1, ... of the CTA (pair): consecutive, so that its hits fall into few partitions
  uint32_t unit, ntl;
  {
    const uint32_t me = PAIR ? (blockIdx.x >> 1) : blockIdx.x, all = PAIR ? (gridDim.x >> 1) : gridDim.x;
    unit = (uint32_t)((uint64_t)n_units * me / all);
    ntl = (uint32_t)((uint64_t)n_units * (me + 1u) / all) - unit;
  }
  auto tile_of = [&](uint32_t u) { return PAIR ? 2u * u + rank : u; };  // this CTA's row tile
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.qt + (PAIR ? rank * qbytes : 0u));
    uint4* dst = reinterpret_cast<uint4*>(sq);
    for (uint32_t i = tid; i < qbytes / 16u; i += blockDim.x) dst[i] = src[i];
    uint4* z = reinterpret_cast<uint4*>(sa);
    for (uint32_t i = tid; i < NB * kTcChunkBytes / 16u; i += blockDim.x) z[i] = make_uint4(0, 0, 0, 0);
    // thresholds as negated FP32 bounds on the score (int keys) or on rowscale * score: every
    // x with key(x) >= th has x >= bound.  With row scales the product is rounded before it becomes
    // a key, and may round up to the threshold, so the bound is the float below it; the exact
    // comparison is made where a hit is appended.
    for (uint32_t i = tid; i < S * Q; i += blockDim.x) {
      const uint32_t p = i / Q, q = i % Q;
      const uint32_t th = q < a.nq ? a.thr[(size_t)(a.q0 + q) * S + p] : 0xFFFFFFFFu;
      float fb;
      if (a.rowscale) {  // x >= +0, key(x) = bits(x) | 2^31; NaN bits: never
        fb = th <= 0x80000000u ? -__int_as_float(0x7f800000)
                               : (th > 0xFF800000u ? __int_as_float(0x7f800000)
                                                   : __uint_as_float((th & 0x7FFFFFFFu) - 1u));
      } else {           // |score| < 2^24, exact in FP32
        const int32_t b = (int32_t)(th ^ 0x80000000u);  // (8-bit filter: below 2^26, rounded down)
        fb = b > (1 << 26) ? __int_as_float(0x7f800000)
                           : (b < -(1 << 26) ? -__int_as_float(0x7f800000) : __int2float_rd(b));
      }
      thf[i] = -fb;
    }
  }
  if (tid == 0) {
    for (uint32_t b = 0; b < kBars; b++) {
      // one arrival per warp; PAIR: both CTAs' epilogues arrive on the even CTA's empty barriers, and
      // the odd CTA's MMA warp once on its staged barriers
      const uint32_t both = PAIR ? 2u : 1u;
      const uint32_t cnt = (b < kDone) ? G / 32 + (PAIR && rank == 0 ? 1u : 0u)
                           : ((b >= kEmpty && b < kDrain) ? both * TcShape<PAIR>::EPI / 32
                           : ((b >= kQueued && b < kDrained) ? TcShape<PAIR>::EPI / 32 : 1u));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(tc_smem_u32(bars + b)), "r"(cnt));
    }
    *gave_up = 0u;
    for (uint32_t b = 0; b < kTcLists; b++) hq_n[b] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kTcMmaWarp) tc_alloc<PAIR>(tc_smem_u32(tslot));
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) tc_cluster_sync();  // both CTAs' barriers exist before any remote arrive
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t b_staged = tc_smem_u32(bars), b_done = tc_smem_u32(bars + kDone);
  const uint32_t b_full = tc_smem_u32(bars + kFull), b_empty = tc_smem_u32(bars + kEmpty);
  const uint32_t b_queued = tc_smem_u32(bars + kQueued), b_drained = tc_smem_u32(bars + kDrained);
  const uint32_t total = ntl * a.nch;  // chunks of this CTA (PAIR: the same in both CTAs)
  bool ok = true;

  if (warp < NB * G / 32u) {
    // ---- producers ----------------------------------------------------------------------------
    // A group of G threads per chunk buffer: group g takes chunks g, g + NB, ...  Its step clears the
    // buffer's last chunk once the MMAs have read it, stages the next one, whose entries were loaded a
    // step earlier, and loads the one after.  A step is a chain of latencies (the wait, the
    // clears, the group's barrier, the stores, the proxy fence: about 1300 cycles, more than a
    // chunk's MMAs), so the groups' steps overlap; the loads come after the hand-over, since the
    // stores would wait for them too.  One group of eight warps for all buffers: 318 us where this
    // takes 290 (2M rows x 1024, 64M entries, 256 queries), 283 and 203 for 128.
    const uint32_t grp = warp / (G / 32u), t = tid - grp * G;
    unsigned char* const ab = sa + grp * kTcChunkBytes;
    // PAIR: the odd CTA's tile of the last unit may lie past the matrix; its chunks are empty
    uint32_t la_i = grp, la_t = tile_of(unit), la_c = grp;
    auto ptr_next = [&](uint32_t& b, uint32_t& e) {  // offsets of chunk la_i, then on to la_i + NB
      while (la_c >= a.nch) {
        la_c -= a.nch;
        la_t += PAIR ? 2u : 1u;
      }
      const bool in = la_i < total && la_t < a.n_rtiles;
      const uint32_t j = la_t * a.nch + la_c;
      b = in ? __ldg(a.ptr + j) : 0u;
      e = in ? __ldg(a.ptr + j + 1) : 0u;
      la_i += NB;
      la_c += NB;
    };
    TcEnt<G> E0, E1;
    uint32_t pb, pe;
    ptr_next(pb, pe);
    E0.load(a.ent, pb, pe - pb, t);
    ptr_next(pb, pe);
    uint32_t j = 0;  // steps done: uses of the buffer
    auto step = [&](TcEnt<G>& cur, TcEnt<G>& old) -> bool {
      if (j > 0) {
        ok &= tc_wait<kAcq>(b_done + 8u * grp, (j - 1u) & 1u, gave_up);
        if (ok) old.stage(ab, a.ent, t, true);
      }
      // every clear lands before any write of this chunk (they may share a byte); the group's
      // threads leave together at the first failure
      if (tc_group_any<G>(grp, !ok)) return false;
      cur.stage(ab, a.ent, t, false);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_arrive_warp<false, true>(b_staged + 8u * grp);
      old.load(a.ent, pb, pe - pb, t);
      ptr_next(pb, pe);
      j++;
      return true;
    };
    bool go = true;
    for (uint32_t i = grp; go && i < total; i += 2u * NB) {
      go = step(E0, E1);
      if (go && i + NB < total) go = step(E1, E0);
    }
    // the odd CTA: before it leaves, the even CTA's commits for its last chunk buffers have landed
    // (those before them were waited for above, those of the accumulators by the epilogue)
    if (PAIR && rank == 1 && t == 0 && go && j > 0) {
      if (!tc_wait_own<kAcq>(b_done + 8u * grp, (j - 1u) & 1u)) *gave_up = 1u;
    }
  } else if (warp >= kTcEpiWarp) {
    // ---- epilogue -----------------------------------------------------------------------------
    const int centre = a.rowstat ? tc_centre(a.qstat) : 0;
    const float qE = a.rowstat ? (float)a.qstat[2] : 0.0f, qQ = a.rowstat ? (float)a.qstat[3] : 0.0f;
    for (uint32_t tl = 0; tl < ntl; tl++) {
      const uint32_t d = tl % ACC;
      const uint32_t T = tile_of(unit + tl), row = tc_epi_row(T);
      // this unit's hit queue is drained of the unit kTcQueues back
      const uint32_t hb = tl % kTcQueues;
      if (tl >= kTcQueues && !a.rowstat) ok &= tc_wait(b_drained + 8u * hb, (tl / kTcQueues - 1u) & 1u, gave_up);
      // without row scales rs = 1: f * 1 is f exactly, so every score takes one path
      const float rs = a.rowscale ? (row < a.n_rows ? __ldg(a.rowscale + row) : 0.0f) : 1.0f;
      const uint2 st = a.rowstat && row < a.n_rows ? __ldg(a.rowstat + row) : make_uint2(0u, 0u);
      tc_prefetch(a, tc_epi_row(tile_of(unit + tl + 1u)));
      const float lim = a.rowstat ? tc_limit(st, centre, qE, qQ, rs) : 0.0f;
      if (ok) ok &= tc_wait<kRlx>(b_full + 8u * d, (tl / ACC) & 1u, gave_up);
      ok = __all_sync(0xFFFFFFFFu, ok);  // tcgen05.ld needs the whole warp
      if (!ok) break;
      tc_fence_after();
      tc_epilogue<PAIR>(a, T, tmem, d, thf, S, rs, lim, b_empty + 8u * d,
                        a.rowstat ? TcQueue{hq_e, hq_n, a.queue_cap}
                                  : TcQueue{hq_e + (size_t)hb * a.queue_cap, hq_n + hb, a.queue_cap});
      if (!a.rowstat) tc_arrive_warp<false, false>(b_queued + 8u * hb);
    }
  } else if (warp >= kTcDrainWarp && warp < kTcDrainWarp + kTcDrains) {
    // ---- drain: the two warps append the queued hits of every other unit, four per lane at a time
    const uint32_t lane = tid & 31u;
    for (uint32_t tl = warp - kTcDrainWarp; tl < ntl && !a.rowstat; tl += kTcDrains) {
      const uint32_t b = tl % kTcQueues, T = tile_of(unit + tl);
      ok = tc_wait(b_queued + 8u * b, (tl / kTcQueues) & 1u, gave_up);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      const uint32_t n = min(*reinterpret_cast<volatile uint32_t*>(hq_n + b), a.queue_cap);
      const volatile uint2* hq = hq_e + (size_t)b * a.queue_cap;
      tc_drain_scores(a, S, hq, n, T);
      __syncwarp();
      if (lane == 0) {
        hq_n[b] = 0u;
        tc_arrive(b_drained + 8u * b);
      }
    }
  } else if (PAIR && warp == kTcMmaWarp && rank == 1) {
    // ---- the odd CTA's staged chunks, passed on to the even CTA (tc_arrive_warp) ----------------
    for (uint32_t i = 0; i < total; i++) {
      const uint32_t buf = i % NB;
      ok = tc_wait(b_staged + 8u * buf, (i / NB) & 1u, gave_up);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      tc_arrive_warp<true, true>(b_staged + 8u * buf);
    }
  } else if (warp == kTcMmaWarp && rank == 0) {
    // ---- MMA issue (one thread of the warp; PAIR: of the even CTA) -----------------------------
    // The warp keeps together but for the issue itself, so that descriptors and addresses are uniform
    // values; a chunk's eight MMAs differ by constants.  Issued from a thread on its own, with the
    // descriptors built for each, an MMA took 122 cycles to issue (now 53), twice what one of 128
    // queries takes to run.
    // instruction descriptor: FP32 accumulator, e4m3 x e4m3, both K-major, N = Q (one CTA: no more
    // than the queries need), M = 128 (256 over a pair)
    const uint32_t n = PAIR ? Q : (min(a.nq, Q) + 15u) & ~15u;
    const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | (((PAIR ? 2u : 1u) * kTcRows >> 4) << 24);
    const uint64_t da0 = tc_desc(tc_smem_u32(sa)), db0 = tc_desc(tc_smem_u32(sq));
    const bool lead = tc_elect();
    uint32_t tl = 0, c = 0, issued = 0;
    for (uint32_t i = 0; i < total && !a.mma_idle; i++) {
      const uint32_t buf = i % NB, d = tl % ACC;
      if (c == 0 && tl >= ACC) ok &= tc_wait<kRlx>(b_empty + 8u * d, ((tl - ACC) / ACC) & 1u, gave_up);
      if (ok) ok &= tc_wait<kAcq>(b_staged + 8u * buf, (i / NB) & 1u, gave_up);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      tc_fence_after();
      const uint32_t nk = min(kTcChunkK, a.kpad - c * kTcChunkK) / 32u;
      const uint64_t da = da0 + buf * (kTcChunkBytes >> 4), db = db0 + c * (kTcChunkBytes >> 4);
      if (lead) {
#pragma unroll
        for (uint32_t kk = 0; kk < kTcChunkK / 32u; kk++)
          if (kk < nk) tc_mma<PAIR>(tmem + d * Q, da + kk * 256u, db + kk * 256u, idesc, (c | kk) != 0);
        tc_commit<PAIR>(b_done + 8u * buf);
        if (c == a.nch - 1) tc_commit<PAIR>(b_full + 8u * d);
      }
      __syncwarp();
      issued = i + 1;
      if (++c == a.nch) {
        c = 0;
        tl++;
      }
    }
    // Before the CTA frees its tensor memory and its shared memory goes away, every MMA this
    // thread issued has completed and the arrivals of its commits have landed, whether the
    // roles finished or gave up: the last commit of each chunk buffer and of each accumulator,
    // and a final commit on the drain barrier (each waited for at most about a second).
    if (issued >= 1) {
      bool drained = true;
      for (uint32_t j = 1; j <= NB && j <= issued; j++)  // the last use of each chunk buffer
        drained &= tc_wait_own<kRlx>(b_done + 8u * ((issued - j) % NB), ((issued - j) / NB) & 1u);
      const uint32_t tiles_full = issued / a.nch;  // units whose accumulator commit was issued
      for (uint32_t j = 1; j <= ACC && j <= tiles_full; j++)  // the last use of each accumulator
        drained &= tc_wait_own<kRlx>(b_full + 8u * ((tiles_full - j) % ACC), ((tiles_full - j) / ACC) & 1u);
      if (lead) tc_commit<PAIR>(tc_smem_u32(bars + kDrain), 1);
      drained &= tc_wait_own<kRlx>(tc_smem_u32(bars + kDrain), 0u);
      if (!drained) *gave_up = 1u;
    }
  }
  tc_fence_before();
  __syncthreads();
  // PAIR: neither CTA frees its tensor memory or leaves while the even CTA's MMAs may still read
  // the odd CTA's shared memory or the odd CTA's roles still arrive on the even CTA's barriers
  if constexpr (PAIR) tc_cluster_sync();
  if (warp == kTcMmaWarp) {
    __syncwarp();
    tc_fence_after();
    tc_dealloc<PAIR>(tmem);
  }
  if (a.rowstat && tid < kTcLists) a.list_n[blockIdx.x * kTcLists + tid] = hq_n[tid];
  if (*gave_up && tid == 0) {
    for (uint32_t q = 0; q < a.nq; q++) atomicOr(a.status + a.q0 + q, ST_DEVICE);
  }
}

}  // namespace dev
}  // namespace aes
