// wtg_bitvec.cu -- rank_support_v<1> and select_support_mcl<1>/<0>
// construction over one bitvector, on the GPU.
//
// One pass over the bitvector (bv_pass_kernel) reads each 512-bit superblock
// once and produces, through a single decoupled look-back scan of the
// superblock one-counts:
//   * the rank_support_v table (rank/rank_support_v_par.hpp:69-123): the
//     absolute count before each superblock (the exclusive scan of :112-113)
//     and the seven 9-bit in-superblock counts (:95-110), including the
//     reference's final-superblock rule (:99-108, and the (total, 0) pair when
//     the capacity is a multiple of 512);
//   * for select_support_mcl, the position of every 64th arg (its
//     superblock starts are every 64th of those) and of every arg that ends a
//     superblock (select_support_mcl_par.hpp:492-523);
// The select structure is then finished per superblock: the long/mini choice
// (span > log^4 n) and widths (:525-543), the pool offsets (a scan), the mini
// blocks from the samples (init_miniblock_serial :440-481), the long blocks by
// re-reading their span (init_longblock_serial :401-438) and m_superblock
// (:546-549).
#include <algorithm>
#include <mutex>

#include "wtg_internal.cuh"
#include "wtg_select.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(bitvec)

constexpr int BV_THREADS = 256;  // one 512-bit superblock per thread

// The pass over the bits.  A tile is SPT * 256 superblocks of 512 bits; the
// tile's one-count is published, the ones before it come from a decoupled
// look-back (word-count scan, no second pass over a count array), and every
// superblock then gets its rank entry and select marks.  Thread per
// superblock: its eight words in four 16-byte loads, popcount prefix and the
// seven 9-bit fields in registers, one 16-byte rank entry.  A warp takes SPT
// runs of 32 consecutive superblocks, so a run's counts are one warp scan.
// With SPT = 4 the words are counted first and read again (from L2, the tile
// is 64 KB) for the marks: a quarter of the look-backs, and few registers
// held across the wait; SPT = 1 keeps a short bitvector on more SMs.
// CTAs are resident and take tiles from a counter, in order.
// One kernel serves every bitvector.  Bound by the integer ALU pipe.  Lanes
// per word (8 to a superblock) with 64-bit arithmetic took 167 us for 842
// Mbit and 226 us for 1.2 Gbit; this takes 83 us for the 842 Mbit (1.3 TB/s
// of bits, 2.3 TB/s with the tables).  Over 21.5 Gbit: 1.78 ms, and 1.58 ms
// where the ones before every superblock were known from the level passes
// (only where n % 512 == 0; the counts cost the build more than that).
//
// Per word, the work is one in-word select at most (the next 64th one or
// zero, see word_marks) in 32-bit arithmetic on per-superblock 64-bit bases:
// the select1 samples of a superblock are consecutive from index
// ceil(ones before / 64), the select0 samples consecutive (descending from
// the back) from ceil(zeros before / 64).  The last two steps of the select
// read a 256 x 8 table of in-byte selects from shared memory.  A superblock
// holds at most one superblock end per polarity (512 < 4096 args), resolved
// once per superblock.  The last superblocks (partial or empty) go word by
// word.
struct SelByteTable {
  uint8_t e[256 * 8];
};
constexpr SelByteTable make_sel_byte_table() {
  SelByteTable t{};
  for (int b = 0; b < 256; ++b) {
    int r = 0;
    for (int k = 0; k < 8; ++k)
      if ((b >> k) & 1) t.e[b * 8 + r++] = (uint8_t)k;
  }
  return t;
}
static __device__ const SelByteTable g_sel_bytes = make_sel_byte_table();

// marks and rank entry of a whole superblock b of words w, sb_before ones before it
__device__ __forceinline__ void superblock_marks(uint64_t b, const uint64_t (&w)[8], uint64_t sb_before, uint32_t flags,
                                                 const uint8_t* __restrict__ lut, uint64_t* __restrict__ rank,
                                                 uint32_t* __restrict__ samples, uint64_t samp_last,
                                                 uint64_t* __restrict__ starts1, uint64_t* __restrict__ starts0,
                                                 uint64_t* __restrict__ ends1, uint64_t* __restrict__ ends0) {
  const bool sel1 = flags & WTG_SELECT1, sel0 = flags & WTG_SELECT0, sel = sel1 || sel0;
  const uint64_t zb = 512 * b - sb_before;  // zeros before the superblock
  const uint32_t pos_base = (uint32_t)(512 * b);
  const uint32_t k1_base = (uint32_t)sb_before, k0_base = (uint32_t)zb;
  // next samples of this superblock: select1 from the front, select0 from the back
  uint32_t* __restrict__ p1 = samples + ((sb_before + 63) >> 6);
  uint32_t* __restrict__ p0 = samples + (samp_last - ((zb + 63) >> 6));
  uint32_t excl = 0;  // ones before the word within the superblock
  uint32_t n1 = 0, n0 = 0;
  uint64_t part = 0;
  uint32_t cnt[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint64_t x = w[j];
    const uint32_t cl = __popc((uint32_t)x);
    const uint32_t cj = cl + __popc((uint32_t)(x >> 32));
    cnt[j] = cj;
    if (j) part |= (uint64_t)excl << (63 - 9 * j);
    if (sel) {
      // branch-free: the select runs for every word, the stores are predicated
      const uint32_t K1 = k1_base + excl;            // ones before the word (mod 2^32)
      const uint32_t K0 = k0_base + 64u * j - excl;  // zeros before it
      const uint32_t d1 = (0u - K1) & 63u, d0 = K1 & 63u;
      const bool s1 = sel1 && d1 < cj, s0 = sel0 && d0 < 64u - cj;
      const uint32_t off = sel64_lut(s1 ? x : ~x, s1 ? d1 : d0, s1 ? cl : 32u - cl, lut);
      // both polarities only when K1 % 64 == 0: the word's first one and first zero
      const uint32_t off0 = s1 ? (uint32_t)(__ffsll((long long)~x) - 1) : off;
      const uint32_t pos = pos_base + 64u * j;
      if (s1) p1[n1] = pos + off;
      if (s0) *(p0 - n0) = pos + off0;
      if (s1 && ((K1 + d1) & 4095u) == 0) starts1[(sb_before + excl + d1) >> 12] = 512 * b + 64 * j + off;
      if (s0 && ((K0 + d0) & 4095u) == 0) starts0[(zb + 64 * j - excl + d0) >> 12] = 512 * b + 64 * j + off0;
      n1 += s1;
      n0 += s0;
    }
    excl += cj;
  }
  if (flags & WTG_RANK) reinterpret_cast<ulonglong2*>(rank)[b] = make_ulonglong2(sb_before, part);
  if (sel) {
    // superblock ends: arg 4095 of a 4096-arg superblock, at most one per
    // polarity in 512 bits; one scan serves the lane's first polarity, the
    // rare superblock that ends one of each takes a second
    const uint32_t cz = 512u - excl;
    const uint32_t e1 = 4095u - (k1_base & 4095u), e0 = 4095u - (k0_base & 4095u);
    bool h1 = sel1 && e1 < excl, h0 = sel0 && e0 < cz;
    while (h1 || h0) {
      const bool t1 = h1;  // this round's polarity
      const uint32_t e = t1 ? e1 : e0;
      uint32_t before = 0, r = 0;
      uint64_t xx = 0, jj = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t cj = t1 ? cnt[j] : 64u - cnt[j];
        const bool here = before <= e && e < before + cj;
        xx = here ? w[j] : xx;
        r = here ? e - before : r;
        jj = here ? (uint64_t)j : jj;
        before += cj;
      }
      xx = t1 ? xx : ~xx;
      const uint64_t pos = 512 * b + 64 * jj + sel64_lut(xx, r, __popc((uint32_t)xx), lut);
      if (t1) ends1[(sb_before + e1) >> 12] = pos;
      else ends0[(zb + e0) >> 12] = pos;
      if (t1) h1 = false;
      else h0 = false;
    }
  }
}

template <int SPT>
__global__ void __launch_bounds__(BV_THREADS)
    bv_pass_kernel(const uint64_t* __restrict__ words, uint64_t size, uint64_t W, uint64_t NB, int vec_ok,
                   uint32_t flags, uint64_t* __restrict__ rank, uint32_t* __restrict__ samples, uint64_t samp_last,
                   uint64_t* __restrict__ starts1, uint64_t* __restrict__ starts0, uint64_t* __restrict__ ends1,
                   uint64_t* __restrict__ ends0, unsigned long long* info, uint64_t* status, uint32_t* counter,
                   uint32_t tile0, uint32_t tile_end, uint32_t* err) {
  constexpr int WARPS = BV_THREADS / 32;
  __shared__ __align__(16) uint8_t lut[256 * 8];  // lut[byte * 8 + r] = position of the r-th set bit of byte
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_wsum[WARPS];
  __shared__ uint64_t s_prefix;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < 128) reinterpret_cast<uint4*>(lut)[tid] = reinterpret_cast<const uint4*>(g_sel_bytes.e)[tid];
  const uint64_t tailmask = (size & 63) ? ((1ull << (size & 63)) - 1) : ~0ull;
  const uint64_t whole = size >> 9;  // superblocks of 512 valid bits; NB, and NB - 1 with a ragged last word, are not
  auto load = [&](uint64_t b, uint64_t(&w)[8]) {  // a whole superblock
    if (vec_ok) {
      const ulonglong2* p = reinterpret_cast<const ulonglong2*>(words + 8 * b);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const ulonglong2 q = __ldg(p + j);
        w[2 * j] = q.x;
        w[2 * j + 1] = q.y;
      }
    } else {  // words not on a 16-byte boundary
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = __ldg(words + 8 * b + j);
    }
  };
  for (;;) {
    __syncthreads();  // the previous tile's shared values are read; the first time, the table is whole
    if (tid == 0) s_tile = tile0 + atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= tile_end) return;
    const uint64_t b0 = (uint64_t)tile * (SPT * BV_THREADS) + warp * (SPT * 32) + lane;
    uint64_t w[8];
    uint32_t ex[SPT];  // ones before the superblock in the warp's run
    uint32_t run = 0;
#pragma unroll
    for (int j = 0; j < SPT; ++j) {
      const uint64_t b = b0 + 32 * j;
      uint32_t c = 0;
      if (b < whole) {
        load(b, w);
#pragma unroll
        for (int k = 0; k < 8; ++k) c += __popcll(w[k]);
      } else if (b <= NB) {
        for (uint64_t wi = 8 * b; wi < W && wi < 8 * b + 8; ++wi) c += __popcll(words[wi] & (wi == W - 1 ? tailmask : ~0ull));
      }
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
      }
      ex[j] = run + inc - c;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_wsum[warp] = run;
    __syncthreads();
    if (warp == 0) {
      const uint32_t v = lane < (uint32_t)WARPS ? s_wsum[lane] : 0u;
      uint32_t inc = v;
#pragma unroll
      for (int o = 1; o < WARPS; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += t;
      }
      if (lane < (uint32_t)WARPS) s_wsum[lane] = inc - v;
      const uint64_t total = __shfl_sync(0xffffffffu, inc, WARPS - 1);
      uint64_t prefix = 0;
      if (tile == 0) {
        if (lane == 0) lb_publish(status, tile, LB_FLAG_INC, total);
      } else {
        if (lane == 0) lb_publish(status, tile, LB_FLAG_AGG, total);
        prefix = lb_lookback_warp(status, tile, err);
        if (lane == 0) lb_publish(status, tile, LB_FLAG_INC, prefix + total);
      }
      if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    const uint64_t before = s_prefix + s_wsum[warp];
#pragma unroll 1
    for (int j = 0; j < SPT; ++j) {
      const uint64_t b = b0 + 32 * j;
      uint32_t e = ex[0];
#pragma unroll
      for (int k = 1; k < SPT; ++k) e = j == k ? ex[k] : e;
      const uint64_t sb_before = before + e;
      if (b < whole) {
        if (SPT > 1) load(b, w);
        superblock_marks(b, w, sb_before, flags, lut, rank, samples, samp_last, starts1, starts0, ends1, ends0);
      } else if (b <= NB) {
        // superblock NB writes fields 1..max(r, 1) of its r words
        // (rank_support_v_par.hpp:99-108); the words' marks one by one
        uint64_t k1 = sb_before, part = 0, lw1 = 0, lw0 = 0;
        const uint64_t r = b < NB ? 7 : W - 8 * NB, kmax = r > 1 ? r : 1;
        for (uint64_t k = 0; k < 8; ++k) {
          const uint64_t wi = 8 * b + k;
          if (k >= 1 && k <= kmax) part |= (k1 - sb_before) << (63 - 9 * k);
          if (wi >= W) continue;
          const uint64_t zmask = wi == W - 1 ? tailmask : ~0ull;
          const uint64_t x = words[wi] & zmask;
          word_marks(x, __popcll(x), k1, wi, zmask, flags & WTG_SELECT1, flags & WTG_SELECT0, samples, samp_last,
                     starts1, starts0, ends1, ends0, lw1, lw0);
          k1 += __popcll(x);
        }
        if (flags & WTG_RANK) {
          rank[2 * b] = sb_before;
          rank[2 * b + 1] = part;
        }
        if (b == NB) {
          info[INF_M1] = k1;
          info[INF_M0] = size - k1;
        }
      }
    }
  }
}

__device__ __forceinline__ uint64_t args_before_sb(int t_b, const uint64_t* __restrict__ rank, uint64_t b) {
  const uint64_t r = rank[2 * b];
  return t_b ? r : 512 * b - r;
}

// position of the last arg, m >= 1: the last superblock with fewer than m
// args before it, found by galloping back from the end over the rank table
// (a dense bitvector ends at the first probe) and a binary search, then its
// words from the last
__device__ uint64_t last_arg_pos(int t_b, const uint64_t* __restrict__ words, const uint64_t* __restrict__ rank,
                                 uint64_t size, uint64_t m) {
  const uint64_t W = (size + 63) >> 6, NB = W >> 3;
  uint64_t lo = NB, hi = NB;
  for (uint64_t step = 1; lo > 0 && args_before_sb(t_b, rank, lo) >= m; step *= 2) {
    hi = lo - 1;
    lo = hi > step ? hi - step : 0;
  }
  while (lo < hi) {
    const uint64_t mid = (lo + hi + 1) >> 1;
    if (args_before_sb(t_b, rank, mid) < m) lo = mid;
    else hi = mid - 1;
  }
  const uint64_t tailmask = (size & 63) ? ((1ull << (size & 63)) - 1) : ~0ull;
  for (uint64_t wi = 8 * lo + 8 < W ? 8 * lo + 8 : W; wi-- > 8 * lo;) {
    uint64_t x = words[wi];
    if (!t_b) x = ~x;
    if (wi == W - 1) x &= tailmask;
    if (x) return (wi << 6) + hi64(x);
  }
  return 0;
}

// The select structures of both polarities, blockIdx.y = t_b.
struct SelBuild {
  const uint64_t* starts;
  const uint64_t* ends;
  uint64_t* descw;      // working descriptors: long flag and width
  uint64_t* offs;       // pool word offset per superblock
  uint64_t* desc;       // final descriptors
  uint64_t* long_list;
  uint64_t* pool;
  uint64_t* sb_words;
  uint64_t* status;     // look-back status words
  uint32_t* counter;
  uint64_t nsb, sb_nwords, m;  // known after the read-back
  uint32_t on;
};
struct SelBuild2 {
  SelBuild t[2];
};

constexpr int SD_THREADS = 256;
constexpr int SD_IPT = 4;  // superblocks per thread, consecutive
constexpr int SD_TILE = SD_THREADS * SD_IPT;

// per superblock: long/mini choice and width (:525-543), and the scan of the
// pool words into offsets in the same launch (decoupled look-back)
__global__ void __launch_bounds__(SD_THREADS)
    select_desc_kernel(SelBuild2 sb2, const uint64_t* __restrict__ words, const uint64_t* __restrict__ rank,
                       uint64_t size, unsigned long long* info, uint64_t logn4, uint32_t* err) {
  __shared__ uint32_t s_tile;
  __shared__ uint64_t s_wsum[SD_THREADS / 32];
  __shared__ uint64_t s_prefix;
  const int t_b = blockIdx.y;
  const SelBuild& sb = sb2.t[t_b];
  if (!sb.on) return;
  const uint64_t m = info[t_b ? INF_M1 : INF_M0];
  const uint64_t nsb = (m + 4095) >> 12;
  if (threadIdx.x == 0) s_tile = atomicAdd(sb.counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((uint64_t)tile * SD_TILE >= nsb) return;  // past the superblocks: no later tile needs this one
  const uint64_t base = (uint64_t)tile * SD_TILE + threadIdx.x * SD_IPT;
  uint32_t sz[SD_IPT];
  uint64_t sum = 0;
#pragma unroll
  for (int k = 0; k < SD_IPT; ++k) {
    const uint64_t i = base + k;
    sz[k] = 0;
    if (i < nsb) {
      const uint64_t start = sb.starts[i];
      uint64_t end;
      if (i + 1 < nsb) {
        end = sb.ends[i];
      } else {
        end = last_arg_pos(t_b, words, rank, size, m);
        info[t_b ? INF_LAST1 : INF_LAST0] = end + 1;
      }
      const uint64_t span = end - start;
      const uint32_t lng = span > logn4;
      const uint32_t wdt = lng ? hi64(end) + 1 : hi64(span) + 1;
      sb.descw[i] = (lng << 7) | wdt;
      sz[k] = lng ? 64 * wdt : wdt;
      if (lng) {
        const unsigned long long slot = atomicAdd(&info[t_b ? INF_NLONG1 : INF_NLONG0], 1ull);
        sb.long_list[slot] = i;
      }
    }
    sum += sz[k];
  }
  uint64_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += t;
  }
  if (lane == 31) s_wsum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const uint64_t v = lane < SD_THREADS / 32 ? s_wsum[lane] : 0;
    uint64_t winc = v;
#pragma unroll
    for (int o = 1; o < SD_THREADS / 32; o <<= 1) {
      const uint64_t t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= (uint32_t)o) winc += t;
    }
    if (lane < SD_THREADS / 32) s_wsum[lane] = winc - v;
    const uint64_t total = __shfl_sync(0xffffffffu, winc, SD_THREADS / 32 - 1);
    uint64_t prefix = 0;
    if (tile == 0) {
      if (lane == 0) lb_publish(sb.status, tile, LB_FLAG_INC, total);
    } else {
      if (lane == 0) lb_publish(sb.status, tile, LB_FLAG_AGG, total);
      prefix = lb_lookback_warp(sb.status, tile, err);
      if (lane == 0) lb_publish(sb.status, tile, LB_FLAG_INC, prefix + total);
    }
    if (lane == 0) s_prefix = prefix;
  }
  __syncthreads();
  uint64_t off = s_prefix + s_wsum[warp] + inc - sum;
#pragma unroll
  for (int k = 0; k < SD_IPT; ++k) {
    const uint64_t i = base + k;
    if (i < nsb) sb.offs[i] = off;
    off += sz[k];
    if (i + 1 == nsb) info[t_b ? INF_POOL1 : INF_POOL0] = off;
  }
}

// The first blocks of each polarity: two superblocks per warp, 16 lanes
// each: final descriptors and the 64-entry mini blocks.  Lane q of a half
// loads entries 4q .. 4q+3 and, for widths of at most 16 (all but sparse
// stretches), packs them into one 64-bit piece at bit 4q * width of the
// block; word q of the block is then two or three pieces fetched by shuffles.
// (Assembling every word from its entries in shared memory took 6-7 loads
// and 64-bit shifts a word and was bound by issue: 0.98 ms of the 2^30 x 20
// build's 5.2 M superblocks, against 0.3 ms of traffic.)  Wider entries go
// word by word through shared memory.  The blocks after them: m_superblock,
// entry i = position of arg 4096*i, width logn.  After an error nothing goes to
// the pool, and the kernels of the long blocks do nothing: the starts and pool
// offsets of a pass whose wait ran out lead out of range.  (The error word is
// tested where the pool is written: before the reads its own read came first in
// every block, 2 us of the 842 Mbit's.)
template <int T_B>
__device__ __forceinline__ void mini_blocks_warp(const SelBuild& sb, uint64_t i0, const uint32_t* __restrict__ samples,
                                                 uint64_t samp_last, uint32_t error, uint32_t (*ent)[64]) {
  const uint32_t lane = threadIdx.x & 31, h = lane >> 4, ql = lane & 15;
  const uint64_t i = i0 + h;
  const bool in = i < sb.nsb;
  // positions are kept mod 2^32; a mini block spans at most log^4 n < 2^32
  // bits, so the offsets are exact
  const uint64_t k0 = 64 * i + 4 * ql;            // first entry's sample
  const uint64_t args = (sb.m + 63) >> 6;         // samples there are
  uint32_t e[4] = {0, 0, 0, 0};
  if (in) {
    if (T_B == 1 && k0 + 4 <= args) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(samples + k0));
      e[0] = v.x, e[1] = v.y, e[2] = v.z, e[3] = v.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k0 + k < args) e[k] = __ldg(samples + (T_B ? k0 + k : samp_last - (k0 + k)));
    }
  }
  uint64_t d = 0, off = 0;
  if (in) {
    d = __ldg(sb.descw + i);
    off = __ldg(sb.offs + i);
    if (ql == 0) sb.desc[i] = (off << 8) | (d & 255);
  }
  const uint32_t start = __shfl_sync(0xffffffffu, e[0], 0, 16);
#pragma unroll
  for (int k = 0; k < 4; ++k) e[k] = k0 + k < args ? e[k] - start : 0u;
  const uint32_t wdt = in && !((d >> 7) & 1) ? (uint32_t)(d & 127) : 0u;  // 0: nothing to pack here
  // entry indices of a word's first and last bit: floor(x / wdt) for
  // x < 2^11 by one multiply with ceil(2^26 / wdt) (exact for x < 2^20,
  // wdt <= 64), not two divisions per word
  const uint64_t rcp = wdt ? ((1u << 26) + wdt - 1) / wdt : 0u;
  if (__any_sync(0xffffffffu, wdt > 16)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) ent[h][4 * ql + k] = e[k];
    __syncwarp();
    for (uint32_t q = ql; q < wdt; q += 16) {
      const uint32_t lo = q * 64;
      const uint32_t j0 = (uint32_t)((lo * rcp) >> 26), j1 = (uint32_t)(((lo + 63) * rcp) >> 26);
      uint64_t out = 0;
      for (uint32_t j = j0; j <= j1 && j < 64; ++j) {
        const uint64_t v = ent[h][j];  // < 2^wdt
        const int32_t sh = (int32_t)(j * wdt) - (int32_t)lo;
        out |= sh >= 0 ? (v << sh) : (v >> (-sh));
      }
      if (!error) sb.pool[off + q] = out;
    }
    return;
  }
  const uint64_t piece = (uint64_t)e[0] | ((uint64_t)e[1] << wdt) | ((uint64_t)e[2] << (2 * wdt)) |
                         ((uint64_t)e[3] << (3 * wdt));
  const uint32_t w4 = 4 * wdt;
  uint32_t j = (uint32_t)((16u * ql * rcp) >> 26);  // piece holding the word's first bit: floor(64 q / w4)
  int32_t sh = (int32_t)(j * w4) - (int32_t)(64 * ql);
  const uint64_t first = __shfl_sync(0xffffffffu, piece, j & 15, 16);
  uint64_t out = wdt ? first >> (-sh) : 0ull;
  for (;;) {
    ++j;
    sh += w4;
    const bool more = wdt && ql < wdt && sh < 64 && j < 16;
    if (!__any_sync(0xffffffffu, more)) break;
    const uint64_t v = __shfl_sync(0xffffffffu, piece, j & 15, 16);
    if (more) out |= v << sh;
  }
  if (ql < wdt && !error) sb.pool[off + ql] = out;
}

__global__ void __launch_bounds__(256)
    select_mini_kernel(SelBuild2 sb2, const uint32_t* __restrict__ samples, uint64_t samp_last, uint32_t logn,
                       const uint32_t* __restrict__ err) {
  __shared__ uint32_t ent[256 / 32][2][64];
  const int t_b = blockIdx.y;
  const SelBuild& sb = sb2.t[t_b];
  if (!sb.on) return;
  const uint32_t error = *err;
  const uint64_t mini_blocks = (sb.nsb + 15) / 16;
  if (blockIdx.x >= mini_blocks) {
    const uint64_t q = (blockIdx.x - mini_blocks) * 256 + threadIdx.x;
    if (q < sb.sb_nwords) sb.sb_words[q] = packed_word(q, logn, sb.nsb, [&](uint64_t i) { return sb.starts[i]; });
    return;
  }
  const uint64_t i0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 2;
  if (i0 >= sb.nsb) return;
  if (t_b) mini_blocks_warp<1>(sb, i0, samples, samp_last, error, ent[threadIdx.x >> 5]);
  else mini_blocks_warp<0>(sb, i0, samples, samp_last, error, ent[threadIdx.x >> 5]);
}

// Long blocks, step 1: the position of every arg of every long superblock,
// one thread per entry (init_longblock_serial, :401-438, restated).  Long
// superblocks are where args are sparse, so instead of scanning their span the
// k-th arg is located by binary search over the rank table's absolute counts
// (between the two samples that bracket it), then within its 512-bit
// superblock by popcounts of at most 8 words.
__global__ void __launch_bounds__(256)
    select_long_fill_kernel(int t_b, const uint64_t* __restrict__ words, uint64_t size, uint64_t W,
                            const uint64_t* __restrict__ rank, const uint64_t* __restrict__ starts,
                            const uint64_t* __restrict__ ends, const unsigned long long* info,
                            const uint64_t* __restrict__ long_list, uint64_t* __restrict__ ent, uint32_t* err) {
  // (uniform over the launch but for an inconsistency that a thread of it reports)
  if (*(volatile const uint32_t*)err) return;
  const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t m = info[t_b ? INF_M1 : INF_M0];
  const uint64_t last = info[t_b ? INF_LAST1 : INF_LAST0];  // last arg position + 1
  const uint64_t nlong = info[t_b ? INF_NLONG1 : INF_NLONG0];
  const uint64_t li = gt >> 12, j = gt & 4095;
  if (li >= nlong) return;
  const uint64_t i = long_list[li];
  const uint64_t k = 4096 * i + j;  // 0-based arg index
  if (k >= m) return;               // entries past the arg count stay zero
  const uint64_t nsb = (m + 4095) >> 12;
  const uint64_t plo = starts[i];
  const uint64_t phi = i + 1 < nsb ? ends[i] : last - 1;
  uint64_t lo = plo >> 9, hi = phi >> 9;  // largest b in [lo, hi] with args_before_sb(b) <= k
  while (lo < hi) {
    const uint64_t mid = (lo + hi + 1) >> 1;
    if (args_before_sb(t_b, rank, mid) <= k) lo = mid;
    else hi = mid - 1;
  }
  uint64_t rem = k - args_before_sb(t_b, rank, lo);
  const uint64_t tailmask = (size & 63) ? ((1ull << (size & 63)) - 1) : ~0ull;
  for (uint64_t wi = 8 * lo; wi < 8 * lo + 8 && wi < W; ++wi) {
    uint64_t x = words[wi];
    if (!t_b) x = ~x;
    if (wi == W - 1) x &= tailmask;
    const uint32_t c = __popcll(x);
    if (rem < c) {
      ent[(li << 12) + j] = (wi << 6) + sel64(x, (uint32_t)rem + 1);
      return;
    }
    rem -= c;
  }
  atomicCAS(err, 0u, (uint32_t)DERR_SELECT_OVERFLOW);  // tables inconsistent
}

// Long blocks, step 2: pack each long block's 4096 positions (width hi(end)+1).
__global__ void __launch_bounds__(256)
    select_long_pack_kernel(int t_b, const unsigned long long* info, const uint64_t* __restrict__ long_list,
                            const uint64_t* __restrict__ descw, const uint64_t* __restrict__ offs,
                            const uint64_t* __restrict__ ent, uint64_t* __restrict__ pool,
                            const uint32_t* __restrict__ err) {
  if (*err) return;
  const uint64_t nlong = info[t_b ? INF_NLONG1 : INF_NLONG0];
  for (uint64_t li = blockIdx.x; li < nlong; li += gridDim.x) {
    const uint64_t i = long_list[li];
    const uint32_t wdt = (uint32_t)(descw[i] & 127);
    const uint64_t off = offs[i];
    const uint64_t* e = ent + li * 4096;
    for (uint64_t q = threadIdx.x; q < 64ull * wdt; q += blockDim.x)
      pool[off + q] = packed_word(q, wdt, 4096, [&](uint64_t j) { return e[j]; });
  }
}

// ------------------------------------------------------------------ host

static uint32_t logn_of(uint64_t size) {
  uint64_t cap = (size + 63) / 64 * 64;
  return hi64(cap) + 1;
}

void bv_release(BvSupport& bv, cudaStream_t s) {
  bv.rank.release(s);
  bv.work.release(s);
  for (auto& sd : bv.sel) {
    sd.sb_words.release(s);
    sd.pool.release(s);
    sd.long_ent.release(s);
  }
}

// superblocks per thread of the pass over a bitvector of NB + 1 superblocks:
// 4 (a 64 KB tile per CTA) once that fills the chip twice, 1 below
static int bv_spt(uint64_t NB) { return NB + 1 >= 4ull * BV_THREADS * 2 * 152 ? 4 : 1; }

int bv_prepare(BvSupport& bv, const uint64_t* d_words, uint64_t size, uint32_t& flags, cudaStream_t s) {
  int rc;
  // select's long blocks are filled through the rank table, so it is built
  // whenever a select support is
  if (flags & (WTG_SELECT1 | WTG_SELECT0)) flags |= WTG_RANK;
  bv.size = size;
  bv.words = d_words;
  bv.flags = flags;
  const uint64_t W = (size + 63) / 64;
  const uint64_t NB = W >> 3;
  const uint64_t nsb_cap = size / 4096 + 2;
  const uint64_t samp_n = W + 2;
  bv.spt = bv_spt(NB);
  const uint64_t tiles = (NB + 1 + bv.spt * BV_THREADS - 1) / (bv.spt * BV_THREADS);
  if (tiles > 0x7fffffffull) return fail(WTG_ERR_INVALID, "bitvector too large");
  bv.tiles = (uint32_t)tiles;
  bv.tiles_done = 0;
  if (flags & WTG_RANK)
    if ((rc = bv.rank.ensure(2 * (NB + 1) * sizeof(uint64_t), s))) return rc;
  DevLayout lay;
  const uint64_t sd_tiles = (nsb_cap + SD_TILE - 1) / SD_TILE;
  const size_t info = lay.add(INF_N * sizeof(uint64_t));
  const size_t status = lay.add((tiles + 1) * sizeof(uint64_t));
  const size_t scan = lay.add(2 * (sd_tiles + 1) * sizeof(uint64_t));
  const size_t clear = lay.bytes;  // these start at 0
  const size_t samples = lay.add(flags & (WTG_SELECT1 | WTG_SELECT0) ? samp_n * sizeof(uint32_t) : 0);
  const size_t per = (nsb_cap * sizeof(uint64_t) + 255) / 256 * 256;
  size_t sel[2] = {0, 0};
  for (int t_b = 0; t_b < 2; ++t_b)
    if (flags & (t_b ? WTG_SELECT1 : WTG_SELECT0)) sel[t_b] = lay.add(6 * per);
  if ((rc = bv.work.ensure(lay.bytes, s))) return rc;
  uint8_t* const w = bv.work.as<uint8_t>();
  WTG_CK(cudaMemsetAsync(w, 0, clear, s));
  bv.info.p = w + info;
  bv.status.p = w + status;
  bv.scan_tmp.p = w + scan;
  bv.samples.p = w + samples;
  for (int t_b = 0; t_b < 2; ++t_b) {
    SelectDev& sd = bv.sel[t_b];
    sd.ends = sd.starts = sd.offs = sd.long_list = sd.desc = DevPart{};
    if (!(flags & (t_b ? WTG_SELECT1 : WTG_SELECT0))) continue;
    uint8_t* const p = w + sel[t_b];
    sd.ends.p = p;
    sd.starts.p = p + per;
    sd.offs.p = p + 2 * per;
    sd.long_list.p = p + 3 * per;
    sd.desc.p = p + 4 * per;  // 2 * nsb_cap entries
  }
  if (test_take_lookback_stall()) {  // tile 0 is never taken: every look-back wait on it runs out
    static const uint32_t one = 1;
    WTG_CK(cudaMemcpyAsync(bv.status.p, &one, sizeof(one), cudaMemcpyHostToDevice, s));
  }
  return WTG_OK;
}

template <int SPT>
static int launch_bv_pass_t(const uint64_t* words, uint64_t size, uint32_t flags, uint64_t* rank, uint32_t* samples,
                            uint64_t samp_last, uint64_t* starts1, uint64_t* starts0, uint64_t* ends1,
                            uint64_t* ends0, unsigned long long* info, uint64_t* status, uint32_t* counter,
                            uint32_t tile0, uint32_t tile_end, uint32_t* err, cudaStream_t s) {
  static const int resident = [] {
    int per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bv_pass_kernel<SPT>, BV_THREADS, 0);
    return std::max(1, per_sm) * std::max(1, sms);
  }();
  const uint64_t W = (size + 63) / 64;
  const unsigned grid = std::min<uint32_t>(tile_end - tile0, (uint32_t)resident);
  prof_begin(PROF_BVPASS, s);
  bv_pass_kernel<SPT><<<grid, BV_THREADS, 0, s>>>(words, size, W, W >> 3, ((uintptr_t)words % 16) == 0, flags, rank,
                                                  samples, samp_last, starts1, starts0, ends1, ends0, info, status,
                                                  counter, tile0, tile_end, err);
  prof_end(PROF_BVPASS, s);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

// every wait of the pass is on a tile taken before, so a launch of at most
// the resident CTAs, or of more, completes
static int launch_bv_pass(int spt, const uint64_t* words, uint64_t size, uint32_t flags, uint64_t* rank,
                          uint32_t* samples, uint64_t samp_last, uint64_t* starts1, uint64_t* starts0,
                          uint64_t* ends1, uint64_t* ends0, unsigned long long* info, uint64_t* status,
                          uint32_t* counter, uint32_t tile0, uint32_t tile_end, uint32_t* err, cudaStream_t s) {
  if (tile_end <= tile0) return WTG_OK;
  auto* const f = spt == 4 ? launch_bv_pass_t<4> : launch_bv_pass_t<1>;
  return f(words, size, flags, rank, samples, samp_last, starts1, starts0, ends1, ends0, info, status, counter, tile0,
           tile_end, err, s);
}

int bv_pass_to(BvSupport& bv, uint64_t bits_ready, uint32_t* d_err, cudaStream_t s) {
  const uint64_t tile_bits = 512ull * BV_THREADS * bv.spt;
  const uint32_t to = bits_ready >= bv.size ? bv.tiles : (uint32_t)(bits_ready / tile_bits);
  // every launch takes its tiles from tiles_done on, counting from 0
  if (bv.tiles_done && to > bv.tiles_done) WTG_CK(cudaMemsetAsync(bv.status.p, 0, sizeof(uint32_t), s));
  const int rc = launch_bv_pass(bv.spt, bv.words, bv.size, bv.flags, bv.rank.as<uint64_t>(),
                                bv.samples.as<uint32_t>(), (bv.size + 63) / 64 + 1, bv.sel[1].starts.as<uint64_t>(),
                                bv.sel[0].starts.as<uint64_t>(), bv.sel[1].ends.as<uint64_t>(),
                                bv.sel[0].ends.as<uint64_t>(), bv.info.as<unsigned long long>(),
                                bv.status.as<uint64_t>() + 1, bv.status.as<uint32_t>(), bv.tiles_done, to, d_err, s);
  if (rc) return rc;
  bv.tiles_done = std::max(bv.tiles_done, to);
  return WTG_OK;
}

uint64_t bv_superblocks_done(const BvSupport& bv) {
  const uint64_t NB = ((bv.size + 63) / 64) >> 3;
  return std::min<uint64_t>(NB + 1, (uint64_t)bv.tiles_done * BV_THREADS * bv.spt);
}

int bv_finish(BvSupport& bv, uint32_t* d_err, cudaStream_t s) {
  int rc;
  const uint32_t flags = bv.flags;
  if (!(flags & (WTG_SELECT1 | WTG_SELECT0))) return WTG_OK;
  const uint64_t size = bv.size;
  const uint64_t W = (size + 63) / 64;
  const uint64_t nsb_cap = size / 4096 + 2;
  const uint64_t samp_n = W + 2;
  const uint32_t logn = logn_of(size);
  const uint64_t logn4 = (uint64_t)(uint32_t)(logn * logn * logn * logn);  // uint32 as in initData
  const uint64_t* d_words = bv.words;
  unsigned long long* info = bv.info.as<unsigned long long>();
  uint32_t* samples = bv.samples.as<uint32_t>();

  // descriptors and pool offsets of both polarities
  const uint64_t tiles = (nsb_cap + SD_TILE - 1) / SD_TILE;
  SelBuild2 sb{};
  for (int t_b = 0; t_b < 2; ++t_b) {
    if (!(flags & (t_b ? WTG_SELECT1 : WTG_SELECT0))) continue;
    SelectDev& sd = bv.sel[t_b];
    SelBuild& x = sb.t[t_b];
    x.on = 1;
    x.starts = sd.starts.as<uint64_t>();
    x.ends = sd.ends.as<uint64_t>();
    x.desc = sd.desc.as<uint64_t>();
    x.descw = x.desc + nsb_cap;
    x.offs = sd.offs.as<uint64_t>();
    x.long_list = sd.long_list.as<uint64_t>();
    x.counter = reinterpret_cast<uint32_t*>(bv.scan_tmp.as<uint64_t>() + t_b * (tiles + 1));
    x.status = bv.scan_tmp.as<uint64_t>() + t_b * (tiles + 1) + 1;
  }
  prof_begin(PROF_SELECT, s);
  select_desc_kernel<<<dim3((unsigned)tiles, 2), SD_THREADS, 0, s>>>(sb, d_words, bv.rank.as<uint64_t>(), size, info,
                                                                     logn4, d_err);
  prof_end(PROF_SELECT, s);
  count_launch();
  WTG_CK(cudaGetLastError());

  // the pool sizes decide the allocations: one small read-back
  uint64_t h[INF_N];
  WTG_CK(cudaMemcpyAsync(h, info, sizeof(h), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));

  uint64_t blocks = 0;
  for (int t_b = 0; t_b < 2; ++t_b) {
    if (!(flags & (t_b ? WTG_SELECT1 : WTG_SELECT0))) continue;
    SelectDev& sd = bv.sel[t_b];
    const uint64_t m = h[t_b ? INF_M1 : INF_M0];
    sd.arg_cnt = m;
    sd.logn = logn;
    sd.logn4 = logn4;
    sd.nsb = (m + 4095) >> 12;
    sd.has_long = h[t_b ? INF_NLONG1 : INF_NLONG0] ? 1 : 0;
    sd.pool_nwords = h[t_b ? INF_POOL1 : INF_POOL0];
    sd.sb_nwords = (sd.nsb * logn + 63) / 64;
    if ((rc = sd.pool.ensure((sd.pool_nwords + 1) * sizeof(uint64_t), s))) return rc;
    if ((rc = sd.sb_words.ensure((sd.sb_nwords + 1) * sizeof(uint64_t), s))) return rc;
    SelBuild& x = sb.t[t_b];
    x.nsb = sd.nsb;
    x.sb_nwords = sd.sb_nwords;
    x.m = m;
    x.pool = sd.pool.as<uint64_t>();
    x.sb_words = sd.sb_words.as<uint64_t>();
    blocks = std::max(blocks, (sd.nsb + 15) / 16 + (sd.sb_nwords + 255) / 256);
  }
  if (blocks) {
    prof_begin(PROF_SELECT, s);
    select_mini_kernel<<<dim3((unsigned)blocks, 2), 256, 0, s>>>(sb, samples, samp_n - 1, logn, d_err);
    prof_end(PROF_SELECT, s);
    count_launch();
    WTG_CK(cudaGetLastError());
  }
  for (int t_b = 0; t_b < 2; ++t_b) {
    const uint64_t nlong = h[t_b ? INF_NLONG1 : INF_NLONG0];
    if (!sb.t[t_b].on || !nlong) continue;
    SelectDev& sd = bv.sel[t_b];
    if ((rc = sd.long_ent.ensure(nlong * 4096 * sizeof(uint64_t), s))) return rc;
    WTG_CK(cudaMemsetAsync(sd.long_ent.p, 0, nlong * 4096 * sizeof(uint64_t), s));
    prof_begin(PROF_SELECT, s);
    select_long_fill_kernel<<<(unsigned)((nlong * 4096 + 255) / 256), 256, 0, s>>>(
        t_b, d_words, size, W, bv.rank.as<uint64_t>(), sd.starts.as<uint64_t>(), sd.ends.as<uint64_t>(), info,
        sd.long_list.as<uint64_t>(), sd.long_ent.as<uint64_t>(), d_err);
    prof_end(PROF_SELECT, s);
    count_launch();
    WTG_CK(cudaGetLastError());
    unsigned grid = (unsigned)std::min<uint64_t>(nlong, 8 * 152);
    prof_begin(PROF_SELECT, s);
    select_long_pack_kernel<<<grid, 256, 0, s>>>(t_b, info, sd.long_list.as<uint64_t>(), sb.t[t_b].descw,
                                                 sb.t[t_b].offs, sd.long_ent.as<uint64_t>(), sd.pool.as<uint64_t>(), d_err);
    prof_end(PROF_SELECT, s);
    count_launch();
    WTG_CK(cudaGetLastError());
  }
  return WTG_OK;
}

int bv_build(BvSupport& bv, const uint64_t* d_words, uint64_t size, uint32_t flags, uint32_t* d_err,
             cudaStream_t s) {
  int rc;
  if ((rc = bv_prepare(bv, d_words, size, flags, s))) return rc;
  if ((rc = bv_pass_to(bv, size, d_err, s))) return rc;
  return bv_finish(bv, d_err, s);
}

// ------------------------------------------------ allocation-free rank build
//
// For callers that must not allocate device memory themselves or through
// this library: code running where the allocator is off limits (inside a
// memory budget owned by another framework, during a phase where cudaMalloc
// would synchronise the device, or on a pool that forbids new allocations).
// The rank pass needs scratch for its look-back status words, its tile
// counter and a few device scalars; here they live in one file-scope device
// array of fixed size, so the call allocates nothing.  Every GPU that loads
// the library holds this array until the process exits.
constexpr uint64_t NOALLOC_MAX_BITS = 1ull << 34;  // 16 Gbit (2 GiB of bits)
constexpr uint64_t NOALLOC_TILES = ((NOALLOC_MAX_BITS >> 9) + 1 + BV_THREADS - 1) / BV_THREADS;
constexpr uint64_t NOALLOC_WORDS = 1 + NOALLOC_TILES + INF_N + 1;  // counter, status, info, error
static __device__ __align__(256) uint64_t g_noalloc_scratch[NOALLOC_WORDS];

static uint64_t* noalloc_scratch_ptr(int dev, int* rc) {
  static std::mutex mu;
  static uint64_t* ptrs[64] = {nullptr};
  if (dev < 0 || dev >= 64) {
    *rc = fail(WTG_ERR_CUDA, "device ordinal out of range");
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(mu);
  // set-up, once per device, with that device current.  The address is kept
  // for the life of the process, so it is not valid after a cudaDeviceReset.
  if (!ptrs[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      *rc = cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
      return nullptr;
    }
    ptrs[dev] = (uint64_t*)p;
  }
  *rc = WTG_OK;
  return ptrs[dev];
}

}  // namespace wtg

extern "C" int wtg_rank_build_noalloc(const uint64_t* d_words, uint64_t size_bits, uint64_t* d_rank,
                                      void* stream) {
  using namespace wtg;
  if ((!d_words && size_bits) || !d_rank) return fail(WTG_ERR_INVALID, "null argument");
  if (size_bits > NOALLOC_MAX_BITS)
    return fail(WTG_ERR_RANGE, "wtg_rank_build_noalloc: size_bits exceeds its fixed scratch (at most 2^34 bits)");
  int dev = 0;
  WTG_CK(cudaGetDevice(&dev));
  int rc;
  uint64_t* scratch = noalloc_scratch_ptr(dev, &rc);
  if (!scratch) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  const uint64_t NB = ((size_bits + 63) / 64) >> 3;
  const int spt = bv_spt(NB);
  const uint64_t tiles = (NB + 1 + spt * BV_THREADS - 1) / (spt * BV_THREADS);
  uint32_t* counter = (uint32_t*)scratch;
  uint64_t* status = scratch + 1;
  unsigned long long* info = (unsigned long long*)(scratch + 1 + NOALLOC_TILES);
  uint32_t* err = (uint32_t*)(scratch + 1 + NOALLOC_TILES + INF_N);
  // the array keeps the previous call's contents: clear what must start at 0
  WTG_CK(cudaMemsetAsync(scratch, 0, (1 + tiles) * sizeof(uint64_t), s));
  WTG_CK(cudaMemsetAsync(info, 0, (INF_N + 1) * sizeof(uint64_t), s));
  if ((rc = launch_bv_pass(spt, d_words, size_bits, WTG_RANK, d_rank, nullptr, 0, nullptr, nullptr, nullptr, nullptr,
                           info, status, counter, 0, (uint32_t)tiles, err, s)))
    return rc;
  // read the error word on the caller's stream only: no device-wide wait
  uint32_t e = 0;
  WTG_CK(cudaMemcpyAsync(&e, err, sizeof(e), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));
  if (e) return fail(WTG_ERR_TIMEOUT, "a device-side wait of the rank pass timed out; the table is invalid");
  return WTG_OK;
}

