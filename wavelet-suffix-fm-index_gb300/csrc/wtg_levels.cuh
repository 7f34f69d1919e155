// wtg_levels.cuh -- the level passes of the tree build (internal): TAU levels
// of the wavelet tree from one read (and, but for the last group, one write)
// of the sequence.
//
// The level-l order is the input stably sorted by the top l bits of each
// symbol, so node p of level l is the range [C_l(p), C_l(p+1)) of it.  A
// group of TAU <= 4 levels l .. l+TAU-1 starts from the level-l order.  Let a
// symbol's digit be its next TAU bits b0 b1 ..; then
//   * bit b_j of symbol i of node p belongs to level l+j at position
//       C_{l+j}(p 2^j + q) + (symbols of p before i with top digit bits q),
//     q = b0 .. b_{j-1};
//   * the symbol's place in the level-(l+TAU) order is
//       C_{l+TAU}(p 2^TAU + d) + (symbols of p before i with digit d).
// With Z_d(i) = symbols before position i with digit d (over the whole
// order, all nodes) the second is base(p, d) + Z_d(i), base(p, d) =
// C_{l+TAU}(p 2^TAU + d) - Z_d(C_l(p)), and the first base_j(p, q) + the sum
// of Z_d(i) over the digits d that start with q.  So a group is three passes:
//   count_kernel       per 1024-symbol chunk its digit counts, scanned over
//                      the chunks in the same launch (decoupled look-back);
//   node_pass_kernel   per node the digit counts before its two ends, from
//                      which the starts and left-child sizes of the next TAU
//                      levels and the record of its bases; and the node of
//                      each chunk's first symbol;
//   level_pass_kernel  the bits of the TAU levels and the scatter.
//
// Symbols lose the bits already used: the order is stored in the narrowest
// of 4, 2 and 1 bytes that holds the remaining bits.  2^30 32-bit symbols
// and 20 levels move 4+4+2 | 2+2+2 | 2+2+1 | 1+1+1 | 1+1 bytes a symbol
// (counted, read, written) where a pass per level moved 8.
//
// All passes work on 32 symbols per lane (a row): a lane reads its row with
// 32-byte loads, gathers the digit's bit planes (one 32-bit word per bit, bit
// i = symbol i), and digit counts are popcounts of masks.  A scattering pass
// takes about 72 warp instructions per 32 symbols for its four levels, where
// a ballot per level and 32 symbols took 36 for each level; it is bound by the
// integer ALU pipe (54-66 %) and shared-memory latency at 15-24 warps per SM
// (two CTAs for 4-byte symbols, three for narrower ones).
// At 2^30 symbols a pass takes 3.5 ms (4 to 2 bytes), 3.0 ms (2 bytes), 2.9
// ms (1 byte), the last one 2.1 ms, the count passes 0.32-0.75 ms; a level
// pass took 1.43 ms before, 19 of them.  Measured and not kept: 32 warps per
// SM (64 registers: spills, 3-5 % slower), the scan of the row counts by
// columns through shared memory (110 instructions fewer a chunk, 4 % slower),
// a swizzled sorted chunk (two instructions a symbol, 5 % slower).
#pragma once
#include <type_traits>

#include "wtg_internal.cuh"

namespace wtg {

constexpr int CHUNK = 1024;  // symbols per warp chunk: 32 rows of 32
constexpr int LOG_CHUNK = 10;
constexpr int LV_THREADS = 256;
constexpr int LV_WARPS = LV_THREADS / 32;
constexpr uint32_t HUFF_OUT = 0xFFFF0000u;  // a Huffman-shaped tree's group passes take up to this many symbols
constexpr int REC = 32;  // words of a node record: bit bases (j, q) at 2^j - 1 + q, scatter bases at 16 + d

// ------------------------------------------------------------------- rows

__device__ __forceinline__ void ld32(const void* p, uint32_t* w) {  // 32 bytes, 32-byte aligned
  uint64_t a, b, c, d;
  asm volatile("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
  w[0] = (uint32_t)a, w[1] = (uint32_t)(a >> 32);
  w[2] = (uint32_t)b, w[3] = (uint32_t)(b >> 32);
  w[4] = (uint32_t)c, w[5] = (uint32_t)(c >> 32);
  w[6] = (uint32_t)d, w[7] = (uint32_t)(d >> 32);
}

// symbols i0 .. i0+31 of src (32-byte aligned, i0 % 32 == 0) as packed words,
// zeros from n on
template <typename T>
__device__ __forceinline__ void load_row(const T* __restrict__ src, uint64_t i0, uint64_t n,
                                         uint32_t (&w)[8 * sizeof(T)]) {
  if (i0 + 32 <= n) {
#pragma unroll
    for (int k = 0; k < (int)sizeof(T); ++k) ld32(reinterpret_cast<const uint8_t*>(src + i0) + 32 * k, w + 8 * k);
  } else {
    constexpr int PER = 4 / sizeof(T);
#pragma unroll
    for (int k = 0; k < 8 * (int)sizeof(T); ++k) {
      uint32_t x = 0;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const uint64_t i = i0 + k * PER + e;
        if (i < n) x |= (uint32_t)__ldg(src + i) << (8 * sizeof(T) * e);
      }
      w[k] = x;
    }
  }
}

// A Huffman-shaped tree's symbols stay bytes; a row of them is taken through
// the group's digit table (shared memory) to 16-bit words, the next four code
// bits above the byte (ds = 8), so that a pass sorts by the digit and stores
// the byte.  3.5 instructions per 32 symbols.
template <typename T, bool HUFF>
__device__ __forceinline__ void load_symbols(const void* __restrict__ src, const uint16_t* s_lut, uint64_t i0,
                                             uint64_t n, uint32_t (&w)[8 * sizeof(T)]) {
  if constexpr (HUFF) {
    uint32_t b[8];
    load_row<uint8_t>(static_cast<const uint8_t*>(src), i0, n, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      w[2 * k] = __byte_perm(s_lut[b[k] & 0xFFu], s_lut[(b[k] >> 8) & 0xFFu], 0x5410);
      w[2 * k + 1] = __byte_perm(s_lut[(b[k] >> 16) & 0xFFu], s_lut[b[k] >> 24], 0x5410);
    }
  } else {
    load_row<T>(static_cast<const T*>(src), i0, n, w);
  }
}

__device__ __forceinline__ void load_lut(const uint16_t* __restrict__ lut, uint16_t* s_lut) {
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_lut[i] = lut[i];
  __syncthreads();
}

// bit planes of the rows' TB-bit digits at bit ds: B[0] the digit's top bit.
// Digits are packed eight to a word first, then each plane is gathered from
// four words at once and put in symbol order by two delta swaps
// (2.6 instructions per 32 symbols and digit for bytes, 3.4 for 16 bits).
template <typename T, int TB>
__device__ __forceinline__ void planes(const uint32_t (&w)[8 * sizeof(T)], int ds, uint32_t (&B)[TB]) {
  uint32_t t[8];  // 4 symbols each, a byte per digit
  if constexpr (sizeof(T) == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = (w[i] >> ds) & 0x0F0F0F0Fu;
  } else if constexpr (sizeof(T) == 2) {
    // symbols 4i, 4i+2, 4i+1, 4i+3 in bytes 0..3
#pragma unroll
    for (int i = 0; i < 8; ++i)
      t[i] = ((w[2 * i] >> ds) & 0x000F000Fu) + (((w[2 * i + 1] >> ds) & 0x000F000Fu) << 8);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t a = __byte_perm(w[4 * i] >> ds, w[4 * i + 1] >> ds, 0x0040);
      const uint32_t b = __byte_perm(w[4 * i + 2] >> ds, w[4 * i + 3] >> ds, 0x0040);
      t[i] = __byte_perm(a, b, 0x5410) & 0x0F0F0F0Fu;
    }
  }
  uint32_t u[4];  // byte b: symbol 8m + b (low nibble) and 8m + 4 + b
#pragma unroll
  for (int m = 0; m < 4; ++m) u[m] = t[2 * m] + (t[2 * m + 1] << 4);
#pragma unroll
  for (int j = 0; j < TB; ++j) {
    uint32_t y = 0;  // bit 8b + 4h + at(m) = symbol 8m + 4h + b
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int at = sizeof(T) == 2 ? ((m & 1) << 1) | (m >> 1) : m;
      const int sh = (TB - 1 - j) - at;
      y |= (sh >= 0 ? u[m] >> sh : u[m] << (-sh)) & (0x11111111u << at);
    }
    uint32_t x;
    if constexpr (sizeof(T) == 2) {  // the two bits of b and of m are exchanged
      x = ((y >> 15) ^ y) & 0x0000AAAAu;
      y ^= x ^ (x << 15);
      x = ((y >> 6) ^ y) & 0x00CC00CCu;
      y ^= x ^ (x << 6);
    } else {
      x = ((y >> 7) ^ y) & 0x00AA00AAu;
      y ^= x ^ (x << 7);
      x = ((y >> 14) ^ y) & 0x0000CCCCu;
      y ^= x ^ (x << 14);
    }
    B[j] = y;
  }
}

// symbols of the row (mask V) with each TB-bit digit, packed two counts to a
// word: digit 2k in the low half of pk[k]
template <int TB>
__device__ __forceinline__ void digit_counts(const uint32_t (&B)[TB], uint32_t V, uint32_t (&pk)[1 << (TB - 1)]) {
  uint32_t m[1 << TB];
  m[0] = V;
#pragma unroll
  for (int j = 0; j < TB; ++j)
#pragma unroll
    for (int q = (1 << j) - 1; q >= 0; --q) {
      m[2 * q + 1] = m[q] & B[j];
      m[2 * q] = m[q] & ~B[j];
    }
#pragma unroll
  for (int k = 0; k < (1 << (TB - 1)); ++k) pk[k] = __popc(m[2 * k]) + ((uint32_t)__popc(m[2 * k + 1]) << 16);
}

// mask of the symbols of row `row` of a chunk that lie in chunk positions [lo, hi)
__device__ __forceinline__ uint32_t row_mask(uint32_t row, uint32_t lo, uint32_t hi) {
  const int32_t a = (int32_t)lo - 32 * (int32_t)row, b = (int32_t)hi - 32 * (int32_t)row;
  const uint32_t below_b = b >= 32 ? 0xFFFFFFFFu : (b <= 0 ? 0u : (1u << b) - 1u);
  const uint32_t below_a = a >= 32 ? 0xFFFFFFFFu : (a <= 0 ? 0u : (1u << a) - 1u);
  return below_b & ~below_a;
}

// ------------------------------------------------------------ node search

// the last p in [lo, hi] with C[p] <= pos (C[lo] <= pos, not decreasing)
__device__ __forceinline__ uint32_t find_node(const uint32_t* __restrict__ C, uint32_t lo, uint32_t hi, uint32_t pos) {
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (__ldg(C + mid) <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------------ count

// A group of levels of a Huffman-shaped tree, whose node sizes are known from
// the byte counts before the build: the records and starts of its first
// level's inner nodes come from the host.  Codes that end inside the group are
// padded with zeros; the strings and children that are not inner nodes are
// left out (word 15 of a record: bit 2^j - 1 + q for string (j, q), bit 16 + d
// for child d).
struct HuffGroup {
  const uint16_t* lut;     // per byte: the group's digit << 8 | byte
  const uint64_t* lv;      // first bit of the group's levels (4), symbols in them (4), symbols of the next group
  const uint32_t* starts;  // of the first level's nodes
  uint32_t* cnode;
  uint32_t nodes;
};

// Digit counts of every chunk and their exclusive scan over the chunks:
// chunkpre[c * 16 + d] = symbols before chunk c with digit d, and the totals
// at c = nchunks.  A CTA takes tiles of 8 * cpw chunks from a counter (so the
// look-back always waits on tiles that have started).  Bound by the read
// of the sequence for 4-byte symbols, by issue for narrower ones.
// HUFF also finds the chunks' nodes (there is no node pass, see HuffGroup).
template <typename T, int TB, bool HUFF = false>
__global__ void __launch_bounds__(LV_THREADS)
    count_kernel(const void* __restrict__ src, uint64_t n, int ds, uint32_t nchunks, int cpw,
                 uint32_t* __restrict__ chunkpre, uint64_t* __restrict__ status, uint32_t sstride,
                 uint32_t* __restrict__ counter, uint32_t tile0, uint32_t tile_end, uint32_t* __restrict__ err,
                 HuffGroup hg) {
  constexpr int MAX_TC = 64;  // chunks per tile
  constexpr int ND = 1 << TB;
  constexpr int NP = 1 << (TB - 1);
  __shared__ __align__(16) uint32_t s_pk[MAX_TC][8];  // per chunk: packed digit counts
  __shared__ uint32_t s_part[16][17];                 // per part of the tile and digit: sums, then prefixes
  __shared__ uint32_t s_tile;
  __shared__ uint16_t s_lut[HUFF ? 256 : 1];
  if constexpr (HUFF) load_lut(hg.lut, s_lut);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tc = LV_WARPS * cpw;
  const uint32_t d = threadIdx.x & 15, part = threadIdx.x >> 4;
  const uint32_t per = (tc + 15) / 16;  // chunks per part
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_tile = tile0 + atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= tile_end) return;
    // narrow symbols two chunks at a time (cpw is 1 or even): both rows are on
    // their way before the first is counted
    constexpr int AHEAD = sizeof(T) == 4 ? 1 : 2;
    for (int k = 0; k < cpw; k += AHEAD) {
      const uint32_t lc = warp * cpw + k;
      const uint32_t c = tile * tc + lc;
      const uint64_t base = (uint64_t)c << LOG_CHUNK;
      uint32_t w[AHEAD][8 * sizeof(T)];
#pragma unroll
      for (int h = 0; h < AHEAD; ++h)
        if (k + h < cpw) load_symbols<T, HUFF>(src, s_lut, base + h * CHUNK + 32 * lane, n, w[h]);  // zeros past the end
#pragma unroll
      for (int h = 0; h < AHEAD; ++h) {
        if (k + h >= cpw) break;
        uint32_t pk[NP], B[TB];
        planes<T, TB>(w[h], ds, B);
        const uint64_t cb = base + h * CHUNK;
        digit_counts<TB>(B, row_mask(lane, 0, cb < n ? (uint32_t)min((uint64_t)CHUNK, n - cb) : 0u), pk);
#pragma unroll
        for (int i = 0; i < NP; ++i) pk[i] = __reduce_add_sync(0xffffffffu, pk[i]);  // halves stay below 2^16
        if (lane == 0) {
#pragma unroll
          for (int i = 0; i < NP; ++i) s_pk[lc + h][i] = pk[i];
        }
      }
    }
    __syncthreads();
    auto count_of = [&](uint32_t lc) -> uint32_t {
      return d < (uint32_t)ND ? (s_pk[lc][d >> 1] >> (16 * (d & 1))) & 0xFFFFu : 0u;
    };
    uint32_t sum = 0;
    for (uint32_t k = 0; k < per; ++k) {
      const uint32_t lc = part * per + k;
      if (lc < tc) sum += count_of(lc);
    }
    s_part[part][d] = sum;
    __syncthreads();
    // warp w: digits 2w (lanes 0-15 hold its parts) and 2w + 1
    {
      const uint32_t dd = 2 * warp + (lane >> 4), pp = lane & 15;
      const uint32_t v = s_part[pp][dd];
      uint32_t inc = v;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o, 16);
        if (pp >= (uint32_t)o) inc += x;
      }
      uint32_t prefix = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t total = __shfl_sync(0xffffffffu, inc, 16 * h + 15);
        const uint32_t dg = 2 * warp + h;
        if (dg >= (uint32_t)ND) continue;
        uint64_t* st = status + (uint64_t)dg * sstride;
        uint64_t before = 0;
        if (tile > 0) {
          if (lane == 0) lb_publish(st, tile, LB_FLAG_AGG, total);
          before = lb_lookback_warp(st, tile, err);
        }
        if (lane == 0) lb_publish(st, tile, LB_FLAG_INC, before + total);
        if ((lane >> 4) == (uint32_t)h) prefix = (uint32_t)before;
      }
      s_part[pp][dd] = prefix + inc - v;
    }
    __syncthreads();
    uint32_t run = s_part[part][d];
    for (uint32_t k = 0; k < per; ++k) {
      const uint32_t lc = part * per + k;
      const uint32_t c = tile * tc + lc;
      if (lc < tc && c < nchunks) {
        chunkpre[(uint64_t)c * 16 + d] = run;
        run += count_of(lc);
        if (c + 1 == nchunks) chunkpre[(uint64_t)nchunks * 16 + d] = run;
      }
    }
    if constexpr (HUFF) {
      for (uint32_t lc = threadIdx.x; lc < tc; lc += LV_THREADS) {
        const uint32_t c = tile * tc + lc;
        if (c < nchunks) {
          hg.cnode[c] = find_node(hg.starts, 0, hg.nodes - 1, c << LOG_CHUNK);
          if (c + 1 == nchunks) hg.cnode[nchunks] = hg.nodes - 1;
        }
      }
    }
  }
}

// ------------------------------------------------------------------ nodes

// Warp per node p of level l: the digit counts before its two ends (chunk
// prefixes plus the counts of the end chunks' heads), then the starts C and
// left-child sizes Z of its descendants on the next TB levels and its record
// (see REC).  Node tables are in heap order: node p of level m at
// 2^m - 1 + p.  Work is a handful of kilobytes a node, latency bound.  Below
// the root, then thread per chunk: the node of its first symbol (neighbours
// search the same way, so their loads coincide).
template <typename T, int TB>
__global__ void __launch_bounds__(LV_THREADS)
    node_pass_kernel(const T* __restrict__ src, uint64_t n, int ds, int l, uint32_t* __restrict__ C,
                     uint32_t* __restrict__ Z, const uint32_t* __restrict__ chunkpre, uint32_t nchunks, int scatter,
                     uint32_t* __restrict__ rec, uint32_t* __restrict__ cnode) {
  constexpr uint32_t ND = 1u << TB;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nodes = 1ull << l;
  const uint64_t stride = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < nodes; p += stride) {
    const uint32_t c0 = l ? C[nodes - 1 + p] : 0u;
    const uint64_t c1 = p + 1 < nodes ? (uint64_t)C[nodes + p] : n;
    // digit counts before position pos, in lanes 0 .. ND-1
    auto before = [&](uint64_t pos) -> uint32_t {
      const uint32_t c = pos >= n ? nchunks : (uint32_t)(pos >> LOG_CHUNK);
      uint32_t z = lane < ND ? __ldg(chunkpre + (uint64_t)c * 16 + lane) : 0u;
      const uint32_t r = c < nchunks ? (uint32_t)(pos & (CHUNK - 1)) : 0u;
      if (r) {  // warp-uniform
        uint32_t w[8 * sizeof(T)], B[TB], pk[ND / 2];
        load_row<T>(src, ((uint64_t)c << LOG_CHUNK) + 32 * lane, n, w);
        planes<T, TB>(w, ds, B);
        digit_counts<TB>(B, row_mask(lane, 0, r), pk);
#pragma unroll
        for (uint32_t k = 0; k < ND / 2; ++k) {
          const uint32_t s = __reduce_add_sync(0xffffffffu, pk[k]);
          if ((lane >> 1) == k) z += (s >> (16 * (lane & 1))) & 0xFFFFu;
        }
      }
      return z;
    };
    uint32_t z0 = 0, size = 0;
    if (c1 > c0) {  // warp-uniform
      z0 = before(c0);
      size = before(c1) - z0;
    }
    uint32_t inc = size, pz = z0;  // scans over the digits
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t a = __shfl_up_sync(0xffffffffu, inc, o), b = __shfl_up_sync(0xffffffffu, pz, o);
      if (lane >= (uint32_t)o) inc += a, pz += b;
    }
    const uint32_t cn = c0 + inc - size;  // start of child `lane` (lane >= ND: the node's end)
    pz -= z0;
    // descendant (j, q) in lane 2^j - 1 + q
    const int j = 31 - __clz(lane + 1);
    const uint32_t q = lane + 1 - (1u << j);
    const bool in = j <= TB;
    const uint32_t a = in ? q << (TB - j) : 0u, b = in ? (q + 1) << (TB - j) : 0u;
    const uint32_t ca = __shfl_sync(0xffffffffu, cn, a);
    const uint32_t mid = __shfl_sync(0xffffffffu, cn, (a + b) >> 1);
    const uint32_t za = __shfl_sync(0xffffffffu, pz, a), zb = __shfl_sync(0xffffffffu, pz, b & 31);
    const uint64_t h = (nodes << j) - 1 + (p << j) + q;
    if (in) {
      if (j || !l) C[h] = ca;  // (below the root the node's own start is there)
      if (j < TB) Z[h] = mid - ca;
    }
    // digit d's scatter base goes to lane 16 + d
    const uint32_t sb = __shfl_sync(0xffffffffu, cn - z0, lane & 15);
    if (c1 > c0) {
      if (lane >= 16) {
        if (scatter) rec[p * REC + lane] = sb;
      } else if (j <= TB) {
        rec[p * REC + lane] = ca - (zb - za);
      }
    }
  }
  if (l) {
    const uint32_t* __restrict__ Cl = C + nodes - 1;
    const uint32_t threads = gridDim.x * blockDim.x;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < nchunks; c += threads)
      cnode[c] = find_node(Cl, 0, (uint32_t)nodes - 1, c << LOG_CHUNK);
    if (blockIdx.x == 0 && threadIdx.x == 0) cnode[nchunks] = (uint32_t)nodes - 1;
  }
}

// ------------------------------------------------------------------- pass

// Shared memory of a warp (byte offsets; a region starts on a 2 KB boundary
// so that addresses are formed by masks):
//   0     slots, 256 bytes per string q of the last level of the group:
//         SCATTER {rank counters of digits 2q, 2q+1 (16 bits each), string},
//         8 bytes a lane; last group the string alone, 4 bytes a lane
//   2048  level 2 of 4: strings, 512 bytes apart, 4 bytes a lane; between
//         them (at 128 of each 512) the level buffers 1..3, and at 128 of the
//         fourth the local digit starts (17 x u16) and scatter deltas
//   4096  SCATTER: the chunk's symbols sorted by digit
template <typename Tin, bool SCATTER>
constexpr uint32_t lv_warp_bytes() {
  return SCATTER ? (4096 + CHUNK * sizeof(Tin) + 2047) / 2048 * 2048 : 4096;
}
template <typename Tin, bool SCATTER>
constexpr uint32_t lv_smem() { return 2048 + LV_WARPS * lv_warp_bytes<Tin, SCATTER>(); }

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void lds64(uint32_t a, uint32_t& x, uint32_t& y) {
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
// ORs v in when it has a bit (lanes with nothing to add would all meet on one word)
__device__ __forceinline__ void ors32(uint32_t a, uint32_t v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %1, 0;\n @p red.shared.or.b32 [%0], %1;\n}\n" ::"r"(a), "r"(v)
               : "memory");
}
// appends the low bit of p at the top of `one` when sel has a bit, else of `zero`
__device__ __forceinline__ void append_to(uint32_t sel, uint32_t p, uint32_t& one, uint32_t& zero) {
  asm("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q shf.r.wrap.b32 %0, %0, %3, 1;\n"
      " @!q shf.r.wrap.b32 %1, %1, %3, 1;\n}\n"
      : "+r"(one), "+r"(zero)
      : "r"(sel), "r"(p));
}
template <typename T>
__device__ __forceinline__ void sts_sym(uint32_t a, uint32_t v) {
  if constexpr (sizeof(T) == 4) asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  else if constexpr (sizeof(T) == 2) asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
  else asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
template <typename T>
__device__ __forceinline__ uint32_t lds_sym(uint32_t a) {
  uint32_t v;
  if constexpr (sizeof(T) == 4) {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  } else if constexpr (sizeof(T) == 2) {
    uint16_t x;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(a) : "memory");
    v = x;
  } else {
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  }
  return v;
}

struct PassArgs {
  const void* src;
  void* dst;
  uint64_t n;
  int ds;         // bit of the digit's lowest bit
  int level;      // the group's first level
  uint32_t nchunks, nodes;
  const uint32_t* Cl;        // starts of the level's nodes
  const uint32_t* chunkpre;  // [nchunks + 1][16]
  const uint32_t* cnode;     // [nchunks + 1] (nodes > 1)
  const uint32_t* rec;       // [nodes][REC]
  uint32_t* bits;
  uint32_t* err;
  HuffGroup huff;  // HUFF passes only
};

// stores the low `take` bits of val, bits [at, at + take) of the bit array
// (take <= 32, at + take within one word)
__device__ __forceinline__ void put_bits(uint32_t* __restrict__ bits, uint64_t word, uint32_t val, uint32_t mask) {
  if (mask == 0xFFFFFFFFu) bits[word] = val;
  else if (val & mask) atomicOr(bits + word, val & mask);
}

// first bit and symbols of the group's level j
template <bool HUFF>
__device__ __forceinline__ uint64_t level_begin(const PassArgs& a, int j) {
  return HUFF ? __ldg(a.huff.lv + j) : (uint64_t)(a.level + j) * a.n;
}
template <bool HUFF>
__device__ __forceinline__ uint64_t level_size(const PassArgs& a, int j) {
  return HUFF ? __ldg(a.huff.lv + 4 + j) : a.n;
}

template <typename Tin, typename Tout, int TAU, bool SCATTER, bool HUFF>
struct LevelPass {
  static constexpr int NW = 8 * sizeof(Tin);
  static constexpr int TB = SCATTER ? TAU : TAU - 1;  // bits that order the strings
  static constexpr int ND = 1 << TB, NP = ND / 2;
  static constexpr int NS = 1 << (TAU - 1);  // strings of the last level
  static constexpr uint32_t QMASK = (NS - 1) << 8;
  static_assert(TAU >= 2 && TAU <= 4 && (!SCATTER || TAU == 4), "");

  static __device__ __forceinline__ uint32_t levelbuf(uint32_t base, int j) {  // words of level j's strings
    return base + 2048 + 512 * (j - 1) + 128 + 4;  // one word of room before
  }

  // appends string acc (its len bits at the top) to level buffer `buf` at bit `off`
  static __device__ __forceinline__ void put(uint32_t buf, uint32_t off, uint32_t acc, uint32_t len) {
    const uint32_t v = __funnelshift_rc(acc, 0u, 32u - len);
    const uint32_t a = buf + ((off >> 5) << 2), sh = off & 31;
    ors32(a, v << sh);
    ors32(a + 4, __funnelshift_l(v, 0u, sh));
  }

  // The symbols V of the rows, all of one node with record word rv (lane r
  // holds word r): their bits of levels 1 .. TAU-1 of the group and their
  // scatter.  zc: in lane d the symbols with digit d before them; on return
  // their own counts are added.  FULL: every symbol of the chunk.
  template <bool FULL>
  static __device__ __forceinline__ void segment(const PassArgs& a, const uint32_t (&w)[NW], const uint32_t (&B)[TAU],
                                                 uint32_t V, uint32_t& zc, uint32_t rv, uint32_t base) {
    const uint32_t lane = threadIdx.x & 31;
    // counts per digit, their scan over the rows, local starts
    uint32_t init[NP], st[NP], own[SCATTER ? 1 : NP];
    {
      uint32_t pk[NP], Bq[TB];
#pragma unroll
      for (int j = 0; j < TB; ++j) Bq[j] = B[j];
      digit_counts<TB>(Bq, V, pk);
#pragma unroll
      for (int k = 0; k < NP; ++k) init[k] = pk[k];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
          const uint32_t x = __shfl_up_sync(0xffffffffu, init[k], o);
          if (lane >= (uint32_t)o) init[k] += x;
        }
      }
      uint32_t run = 0;
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const uint32_t t = __shfl_sync(0xffffffffu, init[k], 31);
        st[k] = run + ((run + (t & 0xFFFFu)) << 16);
        run += (t & 0xFFFFu) + (t >> 16);
        init[k] += st[k] - pk[k];
        if (!SCATTER) own[SCATTER ? 0 : k] = pk[k];
      }
      const uint32_t S = base + 2048 + 512 * 3 + 128;
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NP; ++k) sts32(S + 4 * k, st[k]);
        sts32(S + 4 * NP, run);
      }
    }
    // strings start empty
    const uint32_t sl = base + lane * (SCATTER ? 8 : 4);
    const uint32_t s2 = base + 2048 + lane * 4;
    if constexpr (SCATTER) {
#pragma unroll
      for (int k = 0; k < NP; ++k) sts64(sl + 256 * k, init[k], 0u);
    } else {
#pragma unroll
      for (int q = 0; q < NS; ++q) sts32(sl + 256 * q, 0u);
    }
    if constexpr (TAU == 4) {
#pragma unroll
      for (int q = 0; q < 4; ++q) sts32(s2 + 512 * q, 0u);
    }
#pragma unroll
    for (int j = 1; j < TAU; ++j) {
      sts32(levelbuf(base, j) + 4 * lane, 0u);
      if (lane < 2) sts32(levelbuf(base, j) + 4 * (32 + lane), 0u);
    }
    __syncwarp();
    // symbol by symbol: its bit goes to the end of its string on every level,
    // the symbol to its place in the sorted chunk
    uint32_t a10 = 0, a11 = 0;  // strings of level 1 (TAU > 2)
    {
      uint32_t PL = B[TAU - 1], P2 = B[2 < TAU ? 2 : 0], P1 = B[1];
      const int qs = a.ds + 1 - 8;  // moves the string index to bit 8
      constexpr int PER = 4 / sizeof(Tin);
      int sh[PER];
#pragma unroll
      for (int e = 0; e < PER; ++e) sh[e] = (qs + e * 8 * (int)sizeof(Tin)) & 31;
      const uint32_t stage = base + 4096;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (FULL || ((V >> i) & 1u)) {
          const uint32_t x = w[i / PER];
          const uint32_t rot = __funnelshift_r(x, x, sh[i % PER]);
          const uint32_t as = (rot & QMASK) | sl;
          if constexpr (SCATTER) {
            uint32_t cnt, acc;
            lds64(as, cnt, acc);
            const bool one = rot & 0x80u;
            const uint32_t pos = __byte_perm(cnt, 0u, one ? 0x4432u : 0x4410u);
            cnt += one ? 0x10000u : 1u;
            acc = __funnelshift_r(acc, PL, 1);
            sts64(as, cnt, acc);
            sts_sym<Tin>(stage + pos * (uint32_t)sizeof(Tin), PER == 1 ? x : x >> (8 * sizeof(Tin) * (i % PER)));
          } else {
            sts32(as, __funnelshift_r(lds32(as), PL, 1));
          }
          if constexpr (TAU == 4) {
            const uint32_t a2 = (rot & 0x600u) | s2;
            sts32(a2, __funnelshift_r(lds32(a2), P2, 1));
          }
          if constexpr (TAU > 2) {
            append_to(B[0] & (1u << i), P1, a11, a10);
          }
        }
        PL >>= 1;
        if (TAU == 4) P2 >>= 1;
        if (TAU > 2) P1 >>= 1;
      }
    }
    // the lane's strings into the level buffers
    {
      uint32_t len1[2] = {0, 0}, ex1[2] = {0, 0}, st1[2] = {0, 0};
      uint32_t len2[4] = {0, 0, 0, 0}, ex2[4] = {0, 0, 0, 0}, st2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        uint32_t acc, len, ex, s0;
        if constexpr (SCATTER) {
          uint32_t cnt;
          lds64(sl + 256 * q, cnt, acc);
          const uint32_t o = cnt - init[q], e = init[q] - st[q];
          len = (o & 0xFFFFu) + (o >> 16);
          ex = (e & 0xFFFFu) + (e >> 16);
          s0 = st[q] & 0xFFFFu;
        } else {
          acc = lds32(sl + 256 * q);
          const uint32_t e = init[q / 2] - st[q / 2];
          len = q & 1 ? own[SCATTER ? 0 : q / 2] >> 16 : own[SCATTER ? 0 : q / 2] & 0xFFFFu;
          ex = q & 1 ? e >> 16 : e & 0xFFFFu;
          s0 = q & 1 ? st[q / 2] >> 16 : st[q / 2] & 0xFFFFu;
        }
        put(levelbuf(base, TAU - 1), s0 + ex, acc, len);
        if constexpr (TAU == 4) {
          if (!(q & 1)) st2[q / 2] = s0;
          len2[q / 2] += len;
          ex2[q / 2] += ex;
        }
        if constexpr (TAU > 2) {
          if (q % (NS / 2) == 0) st1[q / (NS / 2)] = s0;
          len1[q / (NS / 2)] += len;
          ex1[q / (NS / 2)] += ex;
        }
      }
      if constexpr (TAU == 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) put(levelbuf(base, 2), st2[q] + ex2[q], lds32(s2 + 512 * q), len2[q]);
      }
      if constexpr (TAU > 2) {
        put(levelbuf(base, 1), st1[0] + ex1[0], a10, len1[0]);
        put(levelbuf(base, 1), st1[1] + ex1[1], a11, len1[1]);
      }
    }
    __syncwarp();
    // lane 2^j - 1 + q: the string (j, q) of the whole segment
    const uint32_t S = base + 2048 + 512 * 3 + 128;
    uint32_t pz = lane < (uint32_t)ND ? zc : 0u;
    const uint32_t z0 = pz;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, pz, o);
      if (lane >= (uint32_t)o) pz += x;
    }
    pz -= z0;
    bool bad = false;
    // (its words of the bitvector, one lane each over all strings of the
    // segment: a string of many words takes no longer than many short ones)
    uint32_t info = 0, glo = 0, ghi = 0, nw = 0;  // info: local start | bits << 11 | level << 22
    {
      const int j = 31 - __clz(lane + 1);
      const uint32_t q = lane + 1 - (1u << j);
      bool in = j >= 1 && j < TAU;
      if constexpr (HUFF) {
        const uint32_t inner = __shfl_sync(0xffffffffu, rv, 15);
        in = in && (inner >> lane & 1u);
      }
      const uint32_t da = in ? q << (TB - j) : 0u, db = in ? (q + 1) << (TB - j) : 0u;
      const uint32_t za = __shfl_sync(0xffffffffu, pz, da), zb = __shfl_sync(0xffffffffu, pz, db);
      if (in) {
        const uint32_t ls = lds16(S + 2 * da);
        const uint32_t len = lds16(S + 2 * db) - ls;
        const uint32_t gp = rv + (zb - za);
        if ((uint64_t)gp + len > level_size<HUFF>(a, j)) {
          bad = true;
        } else if (len) {
          const uint64_t g = level_begin<HUFF>(a, j) + gp;
          glo = (uint32_t)g;
          ghi = (uint32_t)(g >> 32);
          nw = ((glo & 31) + len + 31) >> 5;
          info = ls | (len << 11) | ((uint32_t)j << 22);
        }
      }
    }
    uint32_t wx = nw;  // words of the strings before
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, wx, o);
      if (lane >= (uint32_t)o) wx += x;
    }
    const uint32_t words = __shfl_sync(0xffffffffu, wx, (1 << TAU) - 2);
    wx -= nw;
    for (uint32_t at = 0; at < words; at += 32) {
      const uint32_t i = at + lane;
      uint32_t r = 0;  // the last string with at most i words before it (lane 0 has none: wx = 0)
#pragma unroll
      for (int o = 1 << (TAU - 1); o > 0; o >>= 1) {
        const uint32_t x = __shfl_sync(0xffffffffu, wx, r + o);
        if (r + o < (1u << TAU) - 1 && x <= i) r += o;
      }
      const uint32_t k = i - __shfl_sync(0xffffffffu, wx, r);
      const uint32_t inf = __shfl_sync(0xffffffffu, info, r);
      const uint32_t g0 = __shfl_sync(0xffffffffu, glo, r), g1 = __shfl_sync(0xffffffffu, ghi, r);
      if (i < words) {
        const uint32_t head = g0 & 31, ln = (inf >> 11) & 0x7FFu;
        const int32_t lo = (int32_t)((inf & 0x7FFu) + 32 * k) - (int32_t)head;  // local bit of the word's bit 0
        const uint32_t wa = levelbuf(base, 0) + (inf >> 22) * 512 + (uint32_t)((lo >> 5) * 4);
        const uint32_t val = __funnelshift_r(lds32(wa), lds32(wa + 4), lo & 31);
        uint32_t mask = k == 0 ? 0xFFFFFFFFu << head : 0xFFFFFFFFu;
        const uint32_t end = head + ln - 32 * k;  // valid bits end here
        if (end < 32) mask &= (1u << end) - 1;
        put_bits(a.bits, (((uint64_t)g1 << 32 | g0) >> 5) + k, val, mask);
      }
    }
    if constexpr (SCATTER) {
      const uint32_t s0 = lds16(S + 2 * (lane & 15)), s1 = lds16(S + 2 * ((lane & 15) + 1));
      const uint32_t gd = __shfl_sync(0xffffffffu, rv, 16 + (lane & 15)) + zc;
      const uint64_t next = HUFF ? __ldg(a.huff.lv + 8) : a.n;  // symbols of the next order
      bool goes_on = true;
      if constexpr (HUFF) goes_on = __shfl_sync(0xffffffffu, rv, 15) >> (16 + (lane & 15)) & 1u;
      if (lane < 16) {
        if (goes_on && s1 > s0 && (uint64_t)gd + (s1 - s0) > next) bad = true;
        // (the places of symbols that leave the order come out beyond it)
        sts32(S + 64 + 4 * lane, goes_on ? gd - s0 : HUFF_OUT);
        zc += s1 - s0;
      }
      if (!__any_sync(0xffffffffu, bad)) {
        __syncwarp();
        Tout* __restrict__ dst = static_cast<Tout*>(a.dst);
        const uint32_t total = FULL ? CHUNK : lds16(S + 2 * ND);
        const uint32_t stage = base + 4096;
        const int dsh = a.ds;
#pragma unroll 8
        for (uint32_t r = 0; r < 32; ++r) {
          const uint32_t i = 32 * r + lane;
          if (FULL || i < total) {
            const uint32_t x = lds_sym<Tin>(stage + i * (uint32_t)sizeof(Tin));
            const uint32_t at = i + lds32(S + 64 + (((x >> dsh) & 15u) << 2));
            if (!HUFF || at < next) dst[at] = (Tout)x;
          }
        }
      }
    } else if (!FULL) {
      if (lane < (uint32_t)ND) zc += lds16(S + 2 * (lane + 1)) - lds16(S + 2 * lane);
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicCAS(a.err, 0u, (uint32_t)DERR_BAD_INDEX);
    __syncwarp();
  }

  // A chunk over many small nodes: symbol per lane, row by row, every bit by
  // its own position (counts per string run in shared memory).  Bound by one
  // read after another: the starts of the chunk's nodes are searched in shared
  // memory, and what does not depend on the counts (symbols, nodes, bases) is
  // fetched for four rows at once (10^7 symbols, 20 levels: the passes of levels
  // 12-15 and 16-19 take 69 and 87 us, 87 and 103 row by row).  Bits collected
  // in shared memory before they are set gained nothing.
  static __device__ __noinline__ void scattered_chunk(const PassArgs& a, uint32_t c, uint32_t zc, uint32_t base) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    using Src = typename std::conditional<HUFF, uint8_t, Tin>::type;
    const Src* __restrict__ src = static_cast<const Src*>(a.src);
    // running counts before the row: (j, q) at word 2^j - 1 + q, j = 1 .. TB
    uint32_t pz = lane < (uint32_t)ND ? zc : 0u;
    const uint32_t z0 = pz;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, pz, o);
      if (lane >= (uint32_t)o) pz += x;
    }
    pz -= z0;
    {
      const int j = 31 - __clz(lane + 1);
      const uint32_t q = lane + 1 - (1u << j);
      const bool in = j <= TB;
      const uint32_t da = in ? q << (TB - j) : 0u, db = in ? (q + 1) << (TB - j) : 0u;
      const uint32_t za = __shfl_sync(0xffffffffu, pz, da), zb = __shfl_sync(0xffffffffu, pz, db & 31);
      sts32(base + 4 * lane, in ? zb - za : 0u);
    }
    __syncwarp();
    constexpr int BATCH = 4;
    constexpr uint32_t ROOM = (4096 - 256) / 4;  // node starts that the warp's region holds beside the counts
    const uint32_t p_lo = a.cnode[c], nn = a.cnode[c + 1] - p_lo + 1;
    const bool staged = nn - 1 < ROOM;  // (0 after a count pass's wait that ran out: nodes not in order)
    if (staged) {
      for (uint32_t k = lane; k < nn; k += 32) sts32(base + 256 + 4 * k, __ldg(a.Cl + p_lo + k));
      __syncwarp();
    }
    auto node_of = [&](uint32_t pos) -> uint32_t {
      if (!staged) return find_node(a.Cl, p_lo, p_lo + nn - 1, pos);
      uint32_t lo = 0, hi = nn - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (lds32(base + 256 + 4 * mid) <= pos) lo = mid;
        else hi = mid - 1;
      }
      return p_lo + lo;
    };
    bool bad = false;
    const uint64_t cbase = (uint64_t)c << LOG_CHUNK;
    for (int r0 = 0; r0 < 32 && cbase + 32 * r0 < a.n; r0 += BATCH) {
      uint32_t xs[BATCH], bases[BATCH][TAU], inner[BATCH];  // bases[.][0]: of the scatter
#pragma unroll
      for (int b = 0; b < BATCH; ++b) {
        const uint64_t i = cbase + 32 * (r0 + b) + lane;
        xs[b] = i < a.n ? (uint32_t)src[i] : 0u;
      }
#pragma unroll
      for (int b = 0; b < BATCH; ++b) {
        const uint64_t i = cbase + 32 * (r0 + b) + lane;
        if constexpr (HUFF) xs[b] = __ldg(a.huff.lut + xs[b]);
        const uint32_t dg = (xs[b] >> a.ds) & ((1u << TAU) - 1);
        const uint32_t* __restrict__ rp = a.rec + (uint64_t)(i < a.n ? node_of((uint32_t)i) : p_lo) * REC;
#pragma unroll
        for (int j = 1; j < TAU; ++j) bases[b][j] = __ldg(rp + (1 << j) - 1 + (dg >> (TAU - j)));
        bases[b][0] = SCATTER ? __ldg(rp + 16 + dg) : 0u;
        inner[b] = HUFF ? __ldg(rp + 15) : 0u;
      }
#pragma unroll
      for (int b = 0; b < BATCH; ++b) {
        const uint64_t i = cbase + 32 * (r0 + b) + lane;
        const bool valid = i < a.n;
        const uint32_t x = xs[b];
        const uint32_t dg = (x >> a.ds) & ((1u << TAU) - 1);  // TAU bits
        uint32_t m = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int j = 0; j < TAU; ++j) {
          const bool bit = (dg >> (TAU - 1 - j)) & 1u;
          const uint32_t q = dg >> (TAU - j);  // the j bits above
          if (j >= 1 && valid && (!HUFF || (inner[b] >> ((1 << j) - 1 + q) & 1u))) {
            const uint32_t pos = bases[b][j] + lds32(base + 4 * ((1 << j) - 1 + q)) + __popc(m & lt);
            if (pos >= level_size<HUFF>(a, j)) bad = true;
            else if (bit) {
              const uint64_t g = level_begin<HUFF>(a, j) + pos;
              atomicOr(a.bits + (g >> 5), 1u << (g & 31));
            }
          }
          __syncwarp();
          if (j >= 1 && valid && !(m & ~lt & ~(1u << lane))) {  // the last lane of the string adds its count
            const uint32_t ad = base + 4 * ((1 << j) - 1 + q);
            sts32(ad, lds32(ad) + __popc(m));
          }
          __syncwarp();
          const uint32_t bm = __ballot_sync(0xffffffffu, bit);
          m &= bit ? bm : ~bm;
        }
        if constexpr (SCATTER) {
          if (valid && (!HUFF || (inner[b] >> (16 + dg) & 1u))) {
            const uint32_t pos = bases[b][0] + lds32(base + 4 * (15 + dg)) + __popc(m & lt);
            if (pos >= (HUFF ? __ldg(a.huff.lv + 8) : a.n)) bad = true;
            else static_cast<Tout*>(a.dst)[pos] = (Tout)x;
          }
          __syncwarp();
          if (valid && !(m & ~lt & ~(1u << lane))) {
            const uint32_t ad = base + 4 * (15 + dg);
            sts32(ad, lds32(ad) + __popc(m));
          }
          __syncwarp();
        }
      }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicCAS(a.err, 0u, (uint32_t)DERR_BAD_INDEX);
    __syncwarp();
  }
};

// the group's first level: bit i of the level-l order at level * n + i.
// B0: in each lane the row's word, rows of chunk c, cvalid symbols
__device__ __forceinline__ void first_level_bits(uint32_t* __restrict__ bits, uint64_t g, uint32_t B0,
                                                 uint32_t cvalid) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t head = (uint32_t)(g & 31);
  const uint32_t prev = __shfl_up_sync(0xffffffffu, B0, 1);
  const uint32_t last = __shfl_sync(0xffffffffu, B0, 31);
  const uint64_t G = g >> 5;
  if (head == 0 && cvalid == CHUNK) {
    bits[G + lane] = B0;
    return;
  }
  const uint32_t val = __funnelshift_l(lane ? prev : 0u, B0, head);
  const uint32_t end = head + cvalid;  // bits of the words from G on
  uint32_t mask = 0xFFFFFFFFu;
  if (lane == 0) mask <<= head;
  if (32 * lane < end) {
    if (end - 32 * lane < 32) mask &= (1u << (end - 32 * lane)) - 1;
    put_bits(bits, G + lane, val, mask);
  }
  if (lane == 0 && end > 1024) put_bits(bits, G + 32, last >> (32 - head), (1u << (end - 1024)) - 1);
}

template <typename Tin, typename Tout, int TAU, bool SCATTER, int CTAS, bool HUFF = false>
__global__ void __launch_bounds__(LV_THREADS, CTAS) level_pass_kernel(PassArgs a) {
  using P = LevelPass<Tin, Tout, TAU, SCATTER, HUFF>;
  __shared__ uint16_t s_lut[HUFF ? 256 : 1];
  if constexpr (HUFF) load_lut(a.huff.lut, s_lut);
  extern __shared__ __align__(16) unsigned char lv_smem_raw[];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t base = ((smem_addr(lv_smem_raw) + 2047u) & ~2047u) + warp * lv_warp_bytes<Tin, SCATTER>();
  const uint32_t stride = gridDim.x * LV_WARPS;
  for (uint32_t c = blockIdx.x * LV_WARPS + warp; c < a.nchunks; c += stride) {
    const uint64_t cbase = (uint64_t)c << LOG_CHUNK;
    const uint32_t cvalid = (uint32_t)min((uint64_t)CHUNK, a.n - cbase);
    uint32_t p = 0;
    uint64_t cend = a.n;  // end of the first symbol's node
    if (a.nodes > 1) p = __ldg(a.cnode + c);
    uint32_t zc = lane < (uint32_t)P::ND ? __ldg(a.chunkpre + (uint64_t)c * 16 + lane) : 0u;
    uint32_t w[P::NW], B[TAU];
    load_symbols<Tin, HUFF>(a.src, s_lut, cbase + 32 * lane, a.n, w);
    if (a.nodes > 1 && p + 1 < a.nodes) cend = __ldg(a.Cl + p + 1);
    uint32_t rv = __ldg(a.rec + (uint64_t)p * REC + lane);
    planes<Tin, TAU>(w, a.ds, B);
    first_level_bits(a.bits, level_begin<HUFF>(a, 0) + cbase,
                     cvalid == CHUNK ? B[0] : B[0] & row_mask(lane, 0, cvalid), cvalid);
    if (cend >= cbase + CHUNK && cvalid == CHUNK) {
      P::template segment<true>(a, w, B, 0xFFFFFFFFu, zc, rv, base);
      continue;
    }
    // a few nodes: one after the other; more: symbol by symbol
    if (a.nodes > 1 && __ldg(a.cnode + c + 1) - p > 4) {
      P::scattered_chunk(a, c, zc, base);
      continue;
    }
    uint32_t lo = 0;
    for (;;) {
      const uint32_t hi = (uint32_t)min((uint64_t)cvalid, cend - cbase);
      if (hi > lo) P::template segment<false>(a, w, B, row_mask(lane, lo, hi), zc, rv, base);
      if (hi >= cvalid) break;
      lo = hi;
      ++p;
      cend = p + 1 < a.nodes ? (uint64_t)__ldg(a.Cl + p + 1) : a.n;
      rv = __ldg(a.rec + (uint64_t)p * REC + lane);
    }
  }
}

// a group of one level that is the last: its bits only
template <typename T>
__global__ void __launch_bounds__(LV_THREADS)
    single_level_kernel(const T* __restrict__ src, uint64_t n, int ds, int level, uint32_t nchunks,
                        uint32_t* __restrict__ bits) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * LV_WARPS;
  for (uint32_t c = blockIdx.x * LV_WARPS + (threadIdx.x >> 5); c < nchunks; c += stride) {
    const uint64_t base = (uint64_t)c << LOG_CHUNK;
    const uint32_t cvalid = (uint32_t)min((uint64_t)CHUNK, n - base);
    uint32_t w[8 * sizeof(T)], B[1];
    load_row<T>(src, base + 32 * lane, n, w);
    planes<T, 1>(w, ds, B);
    first_level_bits(bits, (uint64_t)level * n + base, B[0] & row_mask(lane, 0, cvalid), cvalid);
  }
}

}  // namespace wtg
