// wtg_fm_table.cuh -- shared by the backward searches over the balanced and
// the Huffman-shaped tree of a BWT (internal): the interval table of short
// strings and the pattern reader.
#pragma once
#include "wtg_internal.cuh"

namespace wtg {

// Pattern symbols from the back: eight bytes a load, where the aligned eight
// lie inside the patterns' buffer.
struct PatternReader {
  const uint8_t* __restrict__ pat;
  uint64_t total;       // bytes of all patterns
  uint64_t lo = 1ull << 63;  // index of the word in hand (none yet: beyond every index)
  uint64_t word = 0;
  __device__ __forceinline__ PatternReader(const uint8_t* p, uint64_t t) : pat(p), total(t) {}
  __device__ __forceinline__ uint32_t at(uint64_t i) {
    if (i - lo < 8) return (uint32_t)(word >> (8 * (i - lo))) & 255u;
    const uint64_t mis = (uint64_t)(pat + i) & 7;
    if (i >= mis && i - mis + 8 <= total) {
      lo = i - mis;
      word = __ldg(reinterpret_cast<const uint64_t*>(pat + lo));
      return (uint32_t)(word >> (8 * mis)) & 255u;
    }
    return __ldg(pat + i);
  }
};

// Whether a batch of npat patterns over `levels` levels a symbol is worth the
// launches that prepare it (blocks, the table's K, the sort by length: 50 to 90
// us).  Counts of 20 symbols over 2^20 to 2^26 symbols, us without / with: 3
// levels, 2^17 patterns 101-117 / 134-150, 2^18 168-205 / 164-181; 8 levels,
// 2^16 200-273 / 183-272, 2^17 338-416 / 210-333.
inline bool fm_batch_pays(uint64_t npat, uint64_t levels) { return npat * levels >= (3ull << 18); }

// Symbols K of the interval table for a batch: all strings of K symbols have
// at most a quarter of the batch's patterns and 2^19 entries (4 MB of 8-byte
// intervals, a few percent of L2).
inline int fm_table_symbols(uint64_t sigma, uint64_t npat) {
  if (sigma < 2) return 0;
  int K = 0;
  for (uint64_t count = sigma; count <= npat / 4 && count <= (1ull << 19) && K < 19; count *= sigma) ++K;
  return K;
}

// Makes the table (V: an interval) and calls count(K, table); without room
// for it, or where it does not pay, count(0, nullptr).
template <typename V, typename MakeF, typename CountF>
int with_fm_table(bool pays, uint64_t sigma, uint64_t npat, cudaStream_t s, MakeF make, CountF count) {
  const int K = pays ? fm_table_symbols(sigma, npat) : 0;
  if (!K) return count(0, (const V*)nullptr);
  uint64_t entries = 1;
  for (int k = 0; k < K; ++k) entries *= sigma;
  V* const buf = (V*)try_scratch(2 * entries * sizeof(V), s);
  if (!buf) return count(0, (const V*)nullptr);
  // strings of k symbols alternate between the halves and end in the first
  int rc = WTG_OK;
  const V* prev = nullptr;
  uint64_t n = 1;
  for (int k = 1; k <= K && rc == WTG_OK; ++k) {
    V* next = buf + ((K - k) & 1 ? entries : 0);
    rc = make(n, prev, next);
    prev = next;
    n *= sigma;
  }
  if (rc == WTG_OK) rc = count(K, prev);
  cudaFreeAsync(buf, s);
  return rc;
}

}  // namespace wtg
