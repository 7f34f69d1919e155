// wtg_select.cuh -- device-side rank and select over the flat layouts
// (internal; shared by the query kernels and the learned select index).
#pragma once
#include "wtg_internal.cuh"

namespace wtg {

// rank_support_v<1>::rank (rank/rank_support_v_par.hpp:131-142)
__device__ __forceinline__ uint64_t rank1_dev(const uint64_t* __restrict__ tbl, const uint64_t* __restrict__ w,
                                              uint64_t idx) {
  const uint64_t* p = tbl + ((idx >> 8) & 0xFFFFFFFFFFFFFFFEull);
  uint64_t r = p[0] + ((p[1] >> (63 - 9 * ((idx & 0x1FF) >> 6))) & 0x1FF);
  if (idx & 0x3F) r += __popcll(w[idx >> 6] & ((1ull << (idx & 63)) - 1));
  return r;
}

// a rank entry and a word of the bits
__device__ __forceinline__ ulonglong2 load_entry(const uint64_t* __restrict__ rt, uint64_t pos) {
  return __ldg(reinterpret_cast<const ulonglong2*>(rt) + (pos >> 9));
}
__device__ __forceinline__ uint64_t load_word(const uint64_t* __restrict__ words, uint64_t pos) {
  return __ldg(words + (pos >> 6));
}
// ones before pos (mod 2^32) from its rank entry and word
__device__ __forceinline__ uint32_t entry_rank(const ulonglong2& e, uint64_t word, uint64_t pos) {
  const uint32_t in = (uint32_t)(e.y >> (63 - 9 * ((uint32_t)(pos >> 6) & 7))) & 0x1FFu;
  return (uint32_t)e.x + in + __popcll(word & ((1ull << (pos & 63)) - 1));
}

struct SelView {
  const uint64_t* words;
  uint64_t nwords;  // data words at `words`
  const uint64_t* sb_words;
  const uint64_t* desc;
  const uint64_t* pool;
  uint64_t arg_cnt;
  uint32_t logn;
  int has_long;
  int t_b;
};

// The need-th arg (need >= 1) from bit pos on, word by word.  (The first two
// words apart from the rest are the compiler's better code: 2^22 selects over
// 2^30 bits 64 us, 66 in one loop.)
__device__ __forceinline__ uint64_t select_words(const SelView& v, uint64_t pos, uint32_t need) {
  const uint64_t flip = v.t_b ? 0ull : ~0ull;
  uint64_t wp = pos >> 6;
  if (wp >= v.nwords) return NONE64;
  const uint64_t first = (v.words[wp] ^ flip) & (~0ull << (pos & 63));
  uint32_t args = __popcll(first);
  if (args >= need) return (wp << 6) + sel64(first, need);
  uint32_t sum = args;
  if (++wp >= v.nwords) return NONE64;
  uint64_t w = v.words[wp] ^ flip;
  args = __popcll(w);
  while (sum + args < need) {
    sum += args;
    if (++wp >= v.nwords) return NONE64;  // inconsistent tables: never read past the data
    w = v.words[wp] ^ flip;
    args = __popcll(w);
  }
  return (wp << 6) + sel64(w, need - sum);
}

// The same, a sector of four words at a time, one load each, where the words
// start on a sector and the sector lies within them: word by word, every word
// waits for the one before, up to 64 args of a sparse node.
__device__ __forceinline__ uint64_t select_sectors(const SelView& v, uint64_t pos, uint32_t need) {
  if ((uintptr_t)v.words & 31) return select_words(v, pos, need);
  uint64_t wp = pos >> 6;
  const uint64_t flip = v.t_b ? 0ull : ~0ull;
  uint64_t keep = ~0ull << (pos & 63);  // of the first word
  for (uint64_t s = wp & ~3ull; s + 4 <= v.nwords; s += 4) {
    uint64_t w[4];
    asm volatile("ld.global.nc.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(v.words + s));
    uint32_t c[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      w[k] ^= flip;
      if (s + k <= wp) w[k] &= s + k < wp ? 0ull : keep;
      c[k] = __popcll(w[k]);
    }
    const uint32_t c2 = c[0] + c[1], c3 = c2 + c[2], c4 = c3 + c[3];
    if (c4 >= need) {
      const uint32_t k = (c[0] < need) + (c2 < need) + (c3 < need);
      const uint64_t x = k == 0 ? w[0] : k == 1 ? w[1] : k == 2 ? w[2] : w[3];
      const uint32_t before = k == 0 ? 0u : k == 1 ? c[0] : k == 2 ? c2 : c3;
      return ((s + k) << 6) + sel64(x, need - before);
    }
    need -= c4;
    wp = s + 4;  // whole from here on
    keep = ~0ull;
  }
  return select_words(v, (wp << 6) | (keep == ~0ull ? 0 : pos & 63), need);
}

// select_support_mcl::select(i), 1 <= i <= arg_cnt
// (select/select_support_mcl_par.hpp:564-611) on the flat layout; WORDS: see
// select_by_words
template <bool WORDS = false>
__device__ __forceinline__ uint64_t select_dev(const SelView& v, uint64_t i) {
  if (i == 0 || i > v.arg_cnt) return NONE64;
  i = i - 1;
  const uint64_t sb = i >> 12, off = i & 0xFFF;
  const uint64_t d = v.desc[sb];
  const uint32_t wdt = (uint32_t)(d & 127);
  const uint64_t* blk = v.pool + (d >> 8);
  if (v.has_long && ((d >> 7) & 1)) return packed_get(blk, off, wdt);
  const uint64_t base = packed_get(v.sb_words, sb, v.logn);
  const uint64_t mini = packed_get(blk, off >> 6, wdt);
  if ((off & 0x3F) == 0) return base + mini;
  i = i - (sb << 12) - ((off >> 6) << 6);
  const uint64_t pos = base + mini + 1;
  return WORDS ? select_words(v, pos, (uint32_t)i) : select_sectors(v, pos, (uint32_t)i);
}

// Select marks of one 64-bit word wi, given K1 = ones before it: for
// select1 (x) and select0 (~x) the position of every 64th arg (low 32 bits,
// samp[dir * (arg / 64)]), every superblock start (arg 4096q) and end (arg
// 4096q + 4095).  The next multiple of 64 is d1 = (-K1) & 63 ones into the
// word, and d0 = K1 & 63 zeros into it (K0 = 64 wi - K1).  As d1 + d0 is 64
// or 0, a word holds the next 64th arg of at most one polarity unless K1 is
// a multiple of 64, and then both are the word's first one and first zero:
// one branch-free select serves every word.  zmask clears bits past the end.
// lastw1 / lastw0 become wi + 1 when the word holds a one / a zero; a caller
// that visits its words in increasing order turns the final values into
// the position after its last arg with last_arg_end().
__device__ __forceinline__ void word_marks(uint64_t x, uint32_t c, uint64_t K1, uint64_t wi, uint64_t zmask,
                                           bool sel1, bool sel0, uint32_t* __restrict__ samples, uint64_t samp_last,
                                           uint64_t* __restrict__ starts1, uint64_t* __restrict__ starts0,
                                           uint64_t* __restrict__ ends1, uint64_t* __restrict__ ends0,
                                           uint64_t& lastw1, uint64_t& lastw0) {
  const uint64_t z = ~x & zmask;
  const uint32_t cz = __popcll(z);
  const uint64_t K0 = (wi << 6) - K1;
  const uint32_t d1 = (uint32_t)(0u - (uint32_t)K1) & 63u;
  const uint32_t d0 = (uint32_t)K1 & 63u;
  const bool s1 = sel1 && d1 < c, s0 = sel0 && d0 < cz;
  if (s1 || s0) {
    const uint64_t pos = (wi << 6) + sel64_0(s1 ? x : z, s1 ? d1 : d0);
    if (s1) {
      const uint64_t k = K1 + d1;
      samples[k >> 6] = (uint32_t)pos;
      if ((k & 4095) == 0) starts1[k >> 12] = pos;
    }
    if (s0) {
      const uint64_t pos0 = s1 ? (wi << 6) + (uint64_t)(__ffsll((long long)z) - 1) : pos;
      const uint64_t k = K0 + d0;
      samples[samp_last - (k >> 6)] = (uint32_t)pos0;
      if ((k & 4095) == 0) starts0[k >> 12] = pos0;
    }
  }
  if (sel1) {
    const uint32_t e = 4095u - ((uint32_t)K1 & 4095u);
    if (e < c) ends1[(K1 + e) >> 12] = (wi << 6) + sel64_0(x, e);
    lastw1 = c ? wi + 1 : lastw1;
  }
  if (sel0) {
    const uint32_t e = 4095u - ((uint32_t)K0 & 4095u);
    if (e < cz) ends0[(K0 + e) >> 12] = (wi << 6) + sel64_0(z, e);
    lastw0 = cz ? wi + 1 : lastw0;
  }
}

// Position after the last one (t_b = 1) or zero (t_b = 0) of word lastw - 1
// of a bitvector of W words (0 when lastw is 0); read through L2
__device__ __forceinline__ uint64_t last_arg_end(const uint64_t* __restrict__ words, uint64_t lastw, uint64_t W,
                                                 uint64_t tailmask, int t_b) {
  if (!lastw) return 0;
  const uint64_t wi = lastw - 1;
  uint64_t x = __ldcg(words + wi);
  if (!t_b) x = ~x & (wi == W - 1 ? tailmask : ~0ull);
  return (wi << 6) + hi64(x) + 1;
}

// Batches of so many selects hide the latency of reading word by word, and pay
// for what a sector holds beyond the args' word.  (us word by word / by sectors:
// level selects of 2^16 queries, 2^28 x 20 levels, 12.4 / 10.3.)
constexpr uint64_t SEL_MANY = 1ull << 17;
// A bitvector's selects: by words where a word or two hold the arg asked for: in
// such batches where most of the bits are args, in larger ones where a third are
// and L2 holds the bits.  2^22 queries over 2^30 bits, 97 % of them args 56 / 67 us
// (2^18 8.3 / 10.3), half 64 / 68 (2^20 20.9 / 21.0), 3 % 240 / 170; over the levels
// of 2^22 x 20, 64 % args, 71 / 76, 36 % 81 / 84 (2^18 14.5 / 12.4); of 2^28 x 20, 163
// / 154, 131 / 119.
inline bool select_by_words(const SelectDev& sd, uint64_t size, uint64_t nq) {
  if (sd.arg_cnt >= size / 4 * 3) return nq >= SEL_MANY;
  return nq >= 16 * SEL_MANY && sd.arg_cnt >= size / 3 && size / 8 <= (160ull << 20);
}

inline SelView sel_view(const BvSupport& bv, int t_b) {
  const SelectDev& sd = bv.sel[t_b];
  SelView v;
  v.words = bv.words;
  v.nwords = (bv.size + 63) / 64;  // a valid query never reads past the data words
  v.sb_words = sd.sb_words.as<uint64_t>();
  v.desc = sd.desc.as<uint64_t>();
  v.pool = sd.pool.as<uint64_t>();
  v.arg_cnt = sd.arg_cnt;
  v.logn = (uint32_t)sd.logn;
  v.has_long = (int)sd.has_long;
  v.t_b = t_b;
  return v;
}

}  // namespace wtg
