// wtg_fm_table.cuh -- shared by the backward searches over the balanced and
// the Huffman-shaped tree of a BWT (internal): the pattern reader, the plan of a
// large batch and the interval table of short strings.
#pragma once
#include "wtg_blocks.cuh"
#include "wtg_order.cuh"

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

// Large batches are prepared: 192-bit blocks of the tree (wtg_blocks.cuh), a table
// of the intervals of all strings of K symbols, and the patterns taken by length,
// so that the lanes of a warp end together (lengths of 8 to 32 left 48 % of them
// without work).  What of it pays depends on the patterns' lengths, which only
// the device knows: fm_plan_kernel looks at them, and the launches that are not
// wanted do nothing (2.5 us each, 15 us together).
//
// Batches of so many patterns over `levels` levels a symbol are looked at.
// Counts of 20 symbols over 2^20 to 2^26 symbols, us without / with all of it: 3
// levels, 2^17 patterns 101-117 / 134-150, 2^18 168-205 / 164-181; 8 levels, 2^16
// 200-273 / 183-272, 2^17 338-416 / 210-333.
inline bool fm_batch_pays(uint64_t npat, uint64_t levels) { return npat * levels >= (3ull << 18); }

// Most symbols K of the interval table for a batch: all strings of K symbols
// have at most a quarter of the batch's patterns and 2^19 entries (4 MB of 8-byte
// intervals, a few percent of L2).
constexpr int FM_TABLE_MOST = 19;
inline int fm_table_symbols(uint64_t sigma, uint64_t npat) {
  if (sigma < 2) return 0;
  int K = 0;
  for (uint64_t count = sigma; count <= npat / 4 && count <= (1ull << 19) && K < FM_TABLE_MOST; count *= sigma) ++K;
  return K;
}

// a pattern's length, the sort key
struct LengthKey {
  const uint64_t* off;
  __device__ __forceinline__ uint64_t length(uint64_t k) const {
    const uint64_t a = off[k], b = off[k + 1];
    return b > a ? b - a : 0;
  }
  __device__ __forceinline__ uint32_t operator()(uint64_t k) const {
    const uint64_t m = length(k);
    return (uint32_t)(m < 255 ? m : 255);
  }
};

// What of the preparation a batch is worth, from its total length and 1024 of
// its lengths.  A table of the symbols that three quarters of the patterns have
// (a longer one than the patterns was made for nothing: 2^20 patterns of 8
// symbols, 4 letters, 2^24 symbols, 128 us without, 199 with a table of 9).
// Blocks where the symbols left make a dozen probes of each.  Sorting where there
// is enough work left and the longest are longer than the mean.  probes: tree
// positions read a symbol.
constexpr int PLAN_THREADS = 1024;
static __global__ void __launch_bounds__(PLAN_THREADS)
    fm_plan_kernel(LengthKey key, uint64_t npat, int most, uint32_t probes, uint64_t blocks, bool first,
                   uint32_t* __restrict__ flags, uint32_t* __restrict__ hist, uint32_t hist_words) {
  __shared__ uint32_t have[FM_TABLE_MOST + 1];
  __shared__ unsigned long long sum;
  __shared__ uint32_t longest;
  for (uint32_t i = threadIdx.x; i < hist_words; i += PLAN_THREADS) hist[i] = 0;
  if (threadIdx.x == 0) flags[KEYS_DONE] = 0;
  if (!first) return;  // the plan is the call's
  if (threadIdx.x <= FM_TABLE_MOST) have[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    sum = 0;
    longest = 0;
  }
  __syncthreads();
  const uint64_t step = npat >= PLAN_THREADS ? npat / PLAN_THREADS : 1;
  const uint64_t k = min(threadIdx.x * step + (threadIdx.x * 2654435761u) % step, npat - 1);
  const uint32_t len = (uint32_t)min(key.length(k), (uint64_t)0xFFFFFFu);
  atomicAdd(&have[min(len, (uint32_t)most)], 1u);
  const uint32_t all = __reduce_add_sync(0xffffffffu, len), top = __reduce_max_sync(0xffffffffu, len);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sum, (unsigned long long)all);
    atomicMax(&longest, top);
  }
  __syncthreads();
  if (threadIdx.x) return;
  int K = most;
  for (uint32_t n = have[K]; K > 0 && 4 * n < 3 * PLAN_THREADS; n += have[--K]) {
  }
  const uint64_t begin = key.off[0], end = key.off[npat], total = end > begin ? end - begin : 0;
  const uint64_t done = (uint64_t)K * npat, left = (total > done ? total - done : 0) * probes;
  flags[TABLE_SYMBOLS] = K;
  flags[MAKE_BLOCKS] = blocks && left >= 12 * blocks;
  flags[BLOCKS_MADE] = 0;
  flags[AS_IS] = left < 24 * npat || (uint64_t)longest * PLAN_THREADS * 8 <= 9 * sum;
}

// The interval table of a batch, in two launches (each symbol in one of its own
// took up to 19): the strings of up to `first_symbols` symbols, at most 1024, by
// one CTA, the longer ones from those, a thread each.  String c w of k symbols
// lies at c sigma^(k-1) + w.  T: sigma, n, and extend(c, x, y), which prepends
// symbol number c to the interval [x, y).
struct FmTable {
  uint2* first = nullptr;  // sigma^first_symbols entries, the longer strings after them
  int first_symbols = 0;
  uint32_t first_count = 1;
  __device__ __forceinline__ const uint2* of(int K) const { return K > first_symbols ? first + first_count : first; }
};

template <typename T>
__global__ void __launch_bounds__(1024) fm_first_kernel(T t, FmTable table, const uint32_t* __restrict__ flags) {
  __shared__ uint2 s[2][1024];
  const int K = min((int)flags[TABLE_SYMBOLS], table.first_symbols);
  if (!K) return;
  uint32_t count = 1;
  if (threadIdx.x == 0) s[0][0] = make_uint2(0u, (uint32_t)t.n);
  for (int k = 1; k <= K; ++k) {
    __syncthreads();
    const uint32_t i = threadIdx.x, c = i / count;
    if (i < count * t.sigma) {
      uint2 v = s[(k - 1) & 1][i - c * count];
      if (v.x < v.y) t.extend(c, v.x, v.y);
      s[k & 1][i] = v.x < v.y ? v : make_uint2(0u, 0u);
    }
    count *= (uint32_t)t.sigma;
  }
  __syncthreads();
  if (threadIdx.x < count) table.first[threadIdx.x] = s[K & 1][threadIdx.x];
}

template <typename T>
__global__ void __launch_bounds__(256) fm_table_kernel(T t, FmTable table, const uint32_t* __restrict__ flags) {
  const int K = (int)flags[TABLE_SYMBOLS];
  if (K <= table.first_symbols) return;
  uint64_t count = table.first_count;
  for (int k = table.first_symbols; k < K; ++k) count *= t.sigma;
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  uint32_t w = (uint32_t)(i / table.first_count);
  uint2 v = table.first[i - (uint64_t)w * table.first_count];
  for (int k = table.first_symbols; k < K && v.x < v.y; ++k) {
    const uint32_t rest = w / (uint32_t)t.sigma;
    t.extend(w - rest * (uint32_t)t.sigma, v.x, v.y);
    w = rest;
  }
  table.first[table.first_count + i] = v.x < v.y ? v : make_uint2(0u, 0u);
}

// Counts a batch that may be worth it: plans it, makes what the plan wants, and
// calls count(order, table, blocks, first pattern, patterns) for each part of it.
// Without room for the sort: plain() for the whole.  blocks_of: blocks that the
// tree has, 0 where they are not to be made; make_blocks(blocks, wanted).
template <typename T, typename B, typename C, typename P>
int counted_batches(const T& tree, const uint64_t* off, uint64_t npat, uint32_t probes, uint64_t blocks_of,
                    ErrWord& err_word, cudaStream_t own, cudaStream_t s, B make_blocks, C count, P plain) {
  const ErrUse err(err_word, s, own);
  const int most = fm_table_symbols(tree.sigma, npat);
  FmTable table;
  uint4* blocks = nullptr;
  auto key_of = [&](uint64_t at) { return LengthKey{off + at}; };
  const int rc = sorted_batches(
      npat, 0, 1, err.word(), s, key_of,
      [&](uint64_t at, uint64_t, uint32_t* flags, uint32_t* hist, uint32_t words) {
        fm_plan_kernel<<<1, PLAN_THREADS, 0, s>>>(key_of(0), npat, most, probes, blocks_of, at == 0, flags, hist, words);
        count_launch();
      },
      [&](bool sorted, const QueryOrder& o, uint64_t at, uint64_t m) -> int {
        if (!sorted) return plain();
        if (!at) {
          if (blocks_of && (blocks = (uint4*)try_scratch(blocks_of * 32, s)) && !make_blocks(blocks, o.flags + MAKE_BLOCKS))
            return fail(WTG_ERR_CUDA, "pattern blocks: launch failed");
          uint64_t entries = 1;
          for (int k = 0; k < most; ++k) entries *= tree.sigma;
          while (table.first_symbols < most && table.first_count * tree.sigma <= 1024) {
            table.first_count *= (uint32_t)tree.sigma;
            ++table.first_symbols;
          }
          if (most) table.first = (uint2*)try_scratch((table.first_count + entries) * sizeof(uint2), s);
          if (table.first) {
            fm_first_kernel<<<1, 1024, 0, s>>>(tree, table, o.flags);
            count_launch();
            if (most > table.first_symbols) {
              fm_table_kernel<<<(unsigned)((entries + 255) / 256), 256, 0, s>>>(tree, table, o.flags);
              count_launch();
            }
            WTG_CK(cudaGetLastError());
          }
        }
        return count(o, table, blocks, at, m);
      });
  if (table.first) cudaFreeAsync(table.first, s);
  if (blocks) cudaFreeAsync(blocks, s);
  return rc;
}

}  // namespace wtg
