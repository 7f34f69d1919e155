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
#include "wtg_radix.cuh"
#include "wtg_tree.cuh"

namespace wtg {

// After a look-back wait that ran out some places of both hold whatever the
// memory held; a kernel leaves out the ids that are no query of its batch.
struct QueryOrder {
  const uint32_t* pos;  // positions, sorted by their top bits (n: outside the sequence)
  const uint32_t* id;   // the query each belongs to
};

// Queries per sorted batch: bounds the scratch (16 bytes a query, 1 GB) and
// the query numbers.
constexpr uint64_t ORDER_BATCH = 1ull << 26;

static __global__ void __launch_bounds__(256)
    pattern_keys_kernel(const uint64_t* __restrict__ off, uint64_t npat, uint32_t* __restrict__ len) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < npat; k += stride) {
    const uint64_t a = off[k], b = off[k + 1], m = b > a ? b - a : 0;
    len[k] = (uint32_t)(m < 255 ? m : 255);
  }
}

static __global__ void __launch_bounds__(256)
    order_keys_kernel(const uint64_t* __restrict__ q, uint64_t nq, uint64_t n, uint32_t* __restrict__ pos) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nq; k += stride) {
    const uint64_t i = q[k];
    pos[k] = (uint32_t)(i < n ? i : n);
  }
}

// what L2 keeps of a tree: its bits from about 100 MB on (with the rank table 125 MB)
inline bool larger_than_l2(const TreeImpl& t) { return t.n * (uint64_t)t.levels / 8 >= (100ull << 20); }

// When sorting pays: the tree is larger than what L2 keeps of it, has enough
// levels to make up for the sort (60 us, then 10 % of the time) and for reading
// the other arguments by query number, and the batch is large enough.
// Measured, ms as they come / sorted, 2^28 symbols: 20 levels, access of 2^18.5
// queries 0.206 / 0.167, 2^20 0.651 / 0.230, rank 0.155 / 0.167, 0.438 / 0.241;
// 12 levels, access of 2^18.5 0.112 / 0.119, 2^19 0.164 / 0.127, rank 0.111 /
// 0.130; 8 levels, access of 2^19 0.098 / 0.101, 2^19.5 0.141 / 0.110; 3
// levels, 2^24 queries 0.61 / 1.23.  Just above L2 (45 M x 20, 112 MB) access
// of 2^19 0.110 / 0.108, 2^19.5 0.160 / 0.130, rank 0.107 / 0.111, 0.150 /
// 0.134.  Trees that L2 holds gain only by the sectors that neighbours share,
// over many levels: 2^24 x 20, 2^22 queries 0.60 / 0.45, 2^20 queries 0.16 /
// 0.16; 2^25 x 12 0.35 / 0.39.
// Two positions a query (lex_count, range_count) gain from fewer on.
inline bool order_pays(const TreeImpl& t, uint64_t nq, bool two = false) {
  const uint64_t bytes = t.n * (uint64_t)t.levels / 8;
  if (bytes >= (256ull << 20)) return t.levels >= 6 && nq * t.levels >= (two ? 5ull : 7ull) << 20;
  if (larger_than_l2(t)) return t.levels >= 6 && nq >= (5ull << 17);
  return bytes >= (20ull << 20) && t.levels >= 16 && nq >= (1ull << 21);
}

// Sorts the queries of each batch of at most ORDER_BATCH by 8 * passes bits,
// from bit lo on, of the 32-bit keys that make_keys(first, queries, keys)
// writes, and calls launch(true, order, first, queries) for it; without room
// for the scratch launch(false, {}, 0, nq).
template <typename K, typename F>
int sorted_batches(uint64_t nq, int lo, int passes, uint32_t* d_err, cudaStream_t s, K make_keys, F launch) {
  const uint64_t most = nq < ORDER_BATCH ? nq : ORDER_BATCH;
  const uint64_t pairs = (most + 63) / 64 * 64;
  const uint64_t bytes = 16 * pairs + passes * RS_RADIX * 4 + radix_status_bytes(most, passes);
  uint8_t* const scratch = (uint8_t*)try_scratch(bytes, s);
  if (!scratch) return launch(false, QueryOrder{}, 0, nq);  // no room: the queries as they come
  uint32_t* const key[2] = {(uint32_t*)scratch, (uint32_t*)scratch + pairs};
  uint32_t* const val[2] = {(uint32_t*)scratch + 2 * pairs, (uint32_t*)scratch + 3 * pairs};
  uint32_t* hist = (uint32_t*)scratch + 4 * pairs;
  uint8_t* st = (uint8_t*)(hist + passes * RS_RADIX);
  int rc = WTG_OK;
  for (uint64_t at = 0; at < nq && rc == WTG_OK; at += most) {
    const uint64_t m = nq - at < most ? nq - at : most;
    make_keys(at, m, key[0]);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) {
      rc = fail(WTG_ERR_CUDA, "query order: launch failed");
      break;
    }
    int cur = 0;
    rc = radix_sort_pairs<uint32_t>(key, val, m, lo, passes, true, hist, st, d_err, cur, s);
    if (rc == WTG_OK) rc = launch(true, QueryOrder{key[cur], val[cur]}, at, m);
  }
  cudaFreeAsync(scratch, s);
  return rc;
}

// Calls launch(sorted, order, first query, queries) over the batch: sorted by
// position where that pays, otherwise once over all queries as they come.
template <typename F>
int in_order(TreeImpl& t, const uint64_t* pos, uint64_t nq, cudaStream_t s, F launch, bool two = false) {
  if (!order_pays(t, nq, two)) return launch(false, QueryOrder{}, 0, nq);
  constexpr int passes = 2;
  const int bits = 64 - __builtin_clzll(t.n | 1);  // positions 0 .. n
  const ErrUse err(t.err, s, t.stream);
  return sorted_batches(
      nq, bits > 8 * passes ? bits - 8 * passes : 0, passes, err.word(), s,
      [&](uint64_t at, uint64_t m, uint32_t* key) {
        order_keys_kernel<<<(unsigned)((m + 2047) / 2048), 256, 0, s>>>(pos + at, m, t.n, key);
      },
      launch);
}

// Patterns by length (one sort pass), in batches that are worth it: a warp runs
// as long as its longest pattern, and lengths of 8 to 32 left 48 % of the lanes
// without work.
template <typename F>
int by_length(bool pays, const uint64_t* off, uint64_t npat, ErrWord& err_word, cudaStream_t own, cudaStream_t s,
              F launch) {
  if (!pays) return launch(false, QueryOrder{}, 0, npat);
  const ErrUse err(err_word, s, own);
  return sorted_batches(
      npat, 0, 1, err.word(), s,
      [&](uint64_t at, uint64_t m, uint32_t* key) {
        pattern_keys_kernel<<<(unsigned)((m + 2047) / 2048), 256, 0, s>>>(off + at, m, key);
      },
      launch);
}

}  // namespace wtg
