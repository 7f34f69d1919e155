// wtg_order.cuh -- large query batches taken in the order of their positions
// (internal).
//
// A wavelet-tree query reads one rank entry and one word per level, at a
// position that grows with the query's own position inside every node.  In
// the caller's order each of these reads is a trip to DRAM once the tree is
// larger than L2; sorted by the top bits of the position, the queries in
// flight read a narrow window of every node, which stays in L2 and shares
// sectors.  The sort is two 8-bit passes over (position, query number) pairs.
#pragma once
#include <algorithm>

#include "wtg_radix.cuh"
#include "wtg_tree.cuh"

namespace wtg {

// After a look-back wait that ran out some places of both hold whatever the
// memory held; a kernel leaves out the ids that are no query of its batch.
struct QueryOrder {
  const uint32_t* pos;    // positions, sorted by their top bits (n: outside the sequence)
  const uint32_t* id;     // the query each belongs to
  const uint32_t* flags;  // OrderFlags
};

// Words that order_check_kernel or fm_plan_kernel sets: the batch came in the
// order of its positions, or its patterns are of about one length, and nothing of
// the sort has run (pos and id hold nothing); blocks are to be made for it; blocks
// were made for it or for a batch of the call before it; symbols of a pattern
// that the interval table answers.  (KEYS_DONE: CTAs of order_keys_kernel that
// have ended.)
enum OrderFlags { AS_IS = 0, MAKE_BLOCKS, BLOCKS_MADE, KEYS_DONE, TABLE_SYMBOLS, ORDER_FLAGS = 8 };

// the query that thread k takes; false where there is none
__device__ __forceinline__ bool ordered_query(const QueryOrder& ord, uint64_t nq, uint64_t& k) {
  if (!ord.flags[AS_IS]) k = ord.id[k];
  return k < nq;
}

// Queries per sorted batch: bounds the scratch (16 bytes a query, 1 GB) and
// the query numbers.
constexpr uint64_t ORDER_BATCH = 1ull << 26;

// The 32-bit sort key of a query: its position.
struct PositionKey {
  const uint64_t* q;
  uint64_t n;
  __device__ __forceinline__ uint32_t operator()(uint64_t k) const {
    const uint64_t i = q[k];
    return (uint32_t)(i < n ? i : n);
  }
};

// Whether a batch comes in order already (a range read out, a sorted list of
// rows), up or down: of a sample of neighbours none goes the other way by the
// bits that the sort would look at, and next to no two samples.  Such a batch has
// the locality that the sort is for; sorted all the same it took 1.1 to 2.5
// times as long (2^20 consecutive positions, 2^28 symbols x 8 levels, access: 33
// us as they come, 83 sorted).  The launches of the sort and of the blocks do
// nothing then, at about 2.5 us each.  One CTA; it also clears the digit counts.
constexpr int CHECK_THREADS = 1024;
static __global__ void __launch_bounds__(CHECK_THREADS)
    order_check_kernel(PositionKey key, uint64_t nq, int lo, bool first, uint32_t* __restrict__ flags,
                       uint32_t* __restrict__ hist, uint32_t hist_words) {
  for (uint32_t i = threadIdx.x; i < hist_words; i += CHECK_THREADS) hist[i] = 0;
  const uint64_t step = nq >= CHECK_THREADS ? nq / CHECK_THREADS : 1;
  const uint64_t jump = (threadIdx.x * 2654435761u) % (uint32_t)step;  // anywhere in the thread's part
  const uint64_t k = min(threadIdx.x * step + jump, nq - 1);
  const uint32_t a = key(k) >> lo, b = key(min(k + 1, nq - 1)) >> lo, c = key(min(k + step, nq - 1)) >> lo;
  const bool no_up = !__syncthreads_or(b > a), no_down = !__syncthreads_or(b < a);
  const int up = __syncthreads_count(c > a), down = __syncthreads_count(c < a);
  if (threadIdx.x) return;
  constexpr int FEW = CHECK_THREADS / 256;
  const bool as_is = (no_down && down <= FEW) || (no_up && up <= FEW);
  const bool made = !first && flags[BLOCKS_MADE];
  flags[AS_IS] = as_is;
  flags[MAKE_BLOCKS] = !as_is && !made;
  flags[BLOCKS_MADE] = made || !as_is;
  flags[KEYS_DONE] = 0;
}

// Writes the keys of a batch and, in the same pass, clears the sort's status
// words, counts the digits of all its passes and, in the last CTA to end, turns
// the counts into bases (hist: cleared before): what radix_sort_pairs does in two
// memsets and two launches more.
template <typename K>
__global__ void __launch_bounds__(RS_THREADS)
    order_keys_kernel(K make, uint64_t m, int lo, int passes, uint32_t* __restrict__ key, uint32_t* __restrict__ hist,
                      uint4* __restrict__ status, uint64_t status_quads, uint32_t* flags) {
  constexpr int MAX = 2;
  static_assert(MAX * RS_RADIX <= RS_THREADS, "");
  __shared__ uint32_t h[MAX * RS_RADIX];
  __shared__ uint32_t ws[RS_THREADS / 32];
  __shared__ bool s_last;
  if (flags[AS_IS]) return;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < MAX * RS_RADIX) h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t me = (uint64_t)blockIdx.x * RS_THREADS + threadIdx.x, stride = (uint64_t)gridDim.x * RS_THREADS;
  for (uint64_t i = me; i < status_quads; i += stride) status[i] = make_uint4(0u, 0u, 0u, 0u);
  for (uint64_t i = me; i - lane < m; i += stride) {
    const bool in = i < m;
    const uint32_t k = in ? make(i) : 0u;
    if (in) key[i] = k;
    const uint32_t active = __ballot_sync(0xffffffffu, in);
#pragma unroll
    for (int p = 0; p < MAX; ++p) {
      if (p >= passes) break;
      const uint32_t d = ((k >> lo) >> (8 * p)) & 255u;
      int same;
      __match_all_sync(0xffffffffu, d, &same);
      if (same && active == 0xffffffffu) {  // (skewed lengths and repeated positions)
        if (lane == 0) atomicAdd(&h[p * RS_RADIX + d], 32u);
      } else if (in) {
        atomicAdd(&h[p * RS_RADIX + d], 1u);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < passes * RS_RADIX && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], h[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&flags[KEYS_DONE], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // thread: a pass (of 8 warps) and a digit
  const bool on = threadIdx.x < (uint32_t)passes * RS_RADIX;
  const uint32_t v = on ? __ldcg(hist + threadIdx.x) : 0u;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += x;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  for (uint32_t w = warp & ~7u; w < warp; ++w) inc += ws[w];
  if (on) hist[threadIdx.x] = inc - v;
}

// what L2 keeps of a tree: its bits from about 100 MB on (with the rank table 125 MB)
inline bool larger_than_l2(const TreeImpl& t) { return t.n * (uint64_t)t.levels / 8 >= (100ull << 20); }

// When sorting pays: the tree is larger than what L2 keeps of it, has enough
// levels to make up for the sort (45 us, then 10 % of the time) and for reading
// the other arguments by query number, and the batch is large enough.
// Measured, us as they come / sorted, random positions.  2^28 symbols, 20
// levels: access of 2^18.25 queries 152 / 148, 2^18.5 192 / 156, rank 124 / 150,
// 164 / 159, lex_count of 2^18 141 / 159, 2^18.25 160 / 164, range_count 150 / 166,
// 173 / 168, 2^18.5 188 / 170.  12 levels: access of 2^18.5 103 / 110, 2^18.75 121
// / 111, rank of 2^19 113 / 121, 2^19.5 183 / 133, lex_count of 2^18.5 122 / 125,
// 2^18.75 140 / 133, range_count of 2^18.5 140 / 131.  8 levels: access of 2^19 88
// / 94, 2^19.5 131 / 106, rank of 2^19.5 112 / 111, lex_count of 2^19 106 / 116,
// 2^19.3 123 / 132, range_count of 2^19 128 / 124.
// Just above L2 (2^27 x 8, 128 MB): access of 2^19.5 83 / 85, 2^20 117 / 101, rank
// 80 / 88, 107 / 107, lex_count of 2^19.5 108 / 110; 2^28 x 6, rank of 2^20 119 /
// 113, range_count of 2^19.5 135 / 123; 2^26 x 20, access of
// 2^18.75 114 / 99, 2^19.5 205 / 129, rank of 2^19 109 / 110, 2^19.5 159 / 132.
// Trees that L2 holds gain only by the sectors that neighbours share, over many
// levels: 2^24 x 20, 2^21 queries, access 353 / 232, rank 316 / 245.
// two: lex_count and range_count, which read two positions a query.
inline bool order_pays(const TreeImpl& t, uint64_t nq, bool two) {
  const uint64_t bytes = t.n * (uint64_t)t.levels / 8, probes = nq * t.levels;
  if (bytes >= (256ull << 20)) return t.levels >= 6 && probes >= (two ? 6ull : 7ull) << 20;
  if (larger_than_l2(t)) return t.levels >= 6 && nq >= (5ull << 17) && probes >= (two ? 4ull : 8ull) << 20;
  return bytes >= (20ull << 20) && t.levels >= 16 && nq >= (1ull << 21);
}

// Sorts the queries of each batch of at most ORDER_BATCH by 8 * passes bits
// (passes <= 2), from bit lo on, of the keys key_of(first), and calls
// launch(true, order, first, queries) for it; without room for the scratch
// launch(false, {}, 0, nq).  check(first, queries, flags, hist, hist words)
// sets the flags and clears the digit counts.
template <typename K, typename C, typename F>
int sorted_batches(uint64_t nq, int lo, int passes, uint32_t* d_err, cudaStream_t s, K key_of, C check, F launch) {
  const uint64_t most = nq < ORDER_BATCH ? nq : ORDER_BATCH;
  const uint64_t pairs = (most + 63) / 64 * 64;
  const uint32_t hist_words = passes * RS_RADIX;
  const uint64_t status_quads = (radix_status_bytes(most, passes) + 15) / 16;
  uint8_t* const scratch = (uint8_t*)try_scratch(16 * pairs + ORDER_FLAGS * 4 + hist_words * 4 + 16 * status_quads, s);
  if (!scratch) return launch(false, QueryOrder{}, 0, nq);  // no room: the queries as they come
  uint32_t* const key[2] = {(uint32_t*)scratch, (uint32_t*)scratch + pairs};
  uint32_t* const val[2] = {(uint32_t*)scratch + 2 * pairs, (uint32_t*)scratch + 3 * pairs};
  uint32_t* const flags = (uint32_t*)scratch + 4 * pairs;
  uint32_t* const hist = flags + ORDER_FLAGS;
  uint4* const status = (uint4*)(hist + hist_words);
  int rc = WTG_OK;
  for (uint64_t at = 0; at < nq && rc == WTG_OK; at += most) {
    const uint64_t m = nq - at < most ? nq - at : most;
    check(at, m, flags, hist, hist_words);
    const uint64_t ctas = (m + 8 * RS_THREADS - 1) / (8 * RS_THREADS);
    order_keys_kernel<<<(unsigned)(ctas < 152 * 8 ? ctas : 152 * 8), RS_THREADS, 0, s>>>(
        key_of(at), m, lo, passes, key[0], hist, status, status_quads, flags);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) {
      rc = fail(WTG_ERR_CUDA, "query order: launch failed");
      break;
    }
    int cur = 0;
    rc = radix_passes<uint32_t, uint32_t>(key, val, m, lo, passes, true, hist, (uint8_t*)status, d_err, cur, s,
                                          flags + AS_IS);
    if (rc == WTG_OK) rc = launch(true, QueryOrder{key[cur], val[cur], flags}, at, m);
  }
  cudaFreeAsync(scratch, s);
  return rc;
}
static_assert(ORDER_BATCH < (1ull << 30), "32-bit status words");

// Calls launch(sorted, order, first query, queries) over the batch: sorted by
// position where that pays, otherwise once over all queries as they come.
template <typename F>
int in_order(TreeImpl& t, bool two, const uint64_t* pos, uint64_t nq, cudaStream_t s, F launch) {
  if (!order_pays(t, nq, two)) return launch(false, QueryOrder{}, 0, nq);
  constexpr int passes = 2;
  const int bits = 64 - __builtin_clzll(t.n | 1);  // positions 0 .. n
  const int lo = bits > 8 * passes ? bits - 8 * passes : 0;
  const ErrUse err(t.err, s, t.stream);
  auto key_of = [&](uint64_t at) { return PositionKey{pos + at, t.n}; };
  return sorted_batches(
      nq, lo, passes, err.word(), s, key_of,
      [&](uint64_t at, uint64_t m, uint32_t* flags, uint32_t* hist, uint32_t words) {
        order_check_kernel<<<1, CHECK_THREADS, 0, s>>>(key_of(at), m, lo, at == 0, flags, hist, words);
        count_launch();
      },
      launch);
}

}  // namespace wtg
