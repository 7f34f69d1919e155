// wtg_fm.cu -- FM-index counting on the GPU: backward search over the wavelet
// tree of a BWT.
//
// The reference builds the FM-index -- suffix array by divsufsort, the BWT
// s[SA[i]-1] (s[n-1] where SA[i] == 0), a wavelet tree over it
// (fm-index/par/WT.C:33-45) -- and stops there.  Counting is the standard
// backward search: [sp, ep) = [0, n), then for the pattern's symbols from the
// last to the first  sp = C[c] + rank(sp, c),  ep = C[c] + rank(ep, c), where
// rank is wt_int's (wt_int/wt_int_par.hpp:553-577) over the tree of the BWT
// and C[c] counts the symbols below c.
//
// The path of a symbol through the tree does not depend on the position, so
// each symbol's step constants are tabulated once after a build (fm_steps_kernel)
// and kept in shared memory; a rank then costs one rank_support_v probe per
// level, and sp and ep share the path -- and, once the interval is short, the
// rank entry and the word.  Large batches are prepared (wtg_fm_table.cuh): the
// last K symbols of a pattern come from a table of the intervals of all strings
// of K symbols, the others from the tree's bits in 192-bit blocks, and patterns
// of about one length run together.
#include "wtg_fm_table.cuh"
#include "wtg_select.cuh"
#include "wtg_tree.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(fm)

namespace {

// steps[c * L + l]: with x a position of c's node inside level l and R the
// ones before it, bit 0 of c's path goes on at .x + x - R, bit 1 at .y + R
// (mod 2^32; see node_table_kernel); after the last level the result is
// rank(., c)
__global__ void fm_steps_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt, uint64_t n, int L,
                                uint64_t symbols, uint2* __restrict__ steps) {
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= symbols) return;
  uint64_t offset = 0, size = n;
  for (int l = 0; l < L; ++l) {
    const uint64_t o = rank1_dev(rt, tree, offset);
    const uint64_t oe = rank1_dev(rt, tree, offset + size) - o;
    const uint32_t Y = (uint32_t)o, start = (uint32_t)(offset - (uint64_t)l * n);
    const uint32_t zeros = (uint32_t)(size - oe);
    steps[c * L + l] = l + 1 < L ? make_uint2(Y, start + zeros - Y) : make_uint2(Y - start, 0u - Y);
    if ((c >> (L - 1 - l)) & 1) {
      offset += size - oe;
      size = oe;
    } else {
      size -= oe;
    }
    offset += n;
  }
}

// the tree with its rank table, and as 192-bit blocks where they are made
struct FmTree {
  const uint64_t* tree;
  const uint64_t* rt;
  const uint4* blocks;
  const uint2* steps;
  const uint64_t* C;
  uint64_t n, sigma;
  int L;
  // ones before the positions px <= py.  SHARE: what they share is read once,
  // for batches bound by their reads; a small batch waits for its reads, and
  // the second would wait for the first (2^14 patterns: 58 us against 67)
  template <bool BLOCKS, bool SHARE>
  __device__ __forceinline__ void ranks(uint64_t px, uint64_t py, uint32_t& rx, uint32_t& ry) const {
    if constexpr (BLOCKS) {
      uint32_t ox, oy;
      const uint64_t bx = block_of(px, ox), by = block_of(py, oy);
      uint64_t v[4];
      block_load(blocks, bx, v);
      rx = block_at(v, ox).ones;
      if (bx != by) block_load(blocks, by, v);
      ry = block_at(v, oy).ones;
    } else {
      const ulonglong2* __restrict__ re = reinterpret_cast<const ulonglong2*>(rt);
      const ulonglong2 ex = __ldg(re + (px >> 9));
      const uint64_t wx = __ldg(tree + (px >> 6));
      ulonglong2 ey;
      uint64_t wy;
      if constexpr (SHARE) {
        ey = ex;
        wy = wx;
        if ((px ^ py) >> 9) ey = __ldg(re + (py >> 9));
        if ((px ^ py) >> 6) wy = __ldg(tree + (py >> 6));
      } else {
        ey = __ldg(re + (py >> 9));
        wy = __ldg(tree + (py >> 6));
      }
      rx = entry_rank(ex, wx, px);
      ry = entry_rank(ey, wy, py);
    }
  }
  // prepends symbol c (< sigma) to the interval [x, y), but for the C[c] that is
  // not in the steps st
  template <bool BLOCKS, bool SHARE>
  __device__ __forceinline__ void step(const uint2* __restrict__ st, uint32_t c, uint32_t& x, uint32_t& y) const {
    uint64_t lbase = 0;
    for (int l = 0; l < L; ++l, lbase += n) {
      const uint2 s = st[c * L + l];
      uint32_t rx, ry;
      ranks<BLOCKS, SHARE>(lbase + x, lbase + y, rx, ry);
      const bool one = (c >> (L - 1 - l)) & 1;
      x = one ? s.y + rx : s.x + x - rx;
      y = one ? s.y + ry : s.x + y - ry;
    }
  }
  __device__ __forceinline__ void extend(uint32_t c, uint32_t& x, uint32_t& y) const {
    const uint32_t base = (uint32_t)__ldg(C + c);
    step<false, true>(steps, c, x, y);
    x += base;
    y += base;
  }
  // bytes of a CTA's steps in shared memory: at most 256 symbols x 24 levels
  size_t shared_bytes() const { return sigma * L * sizeof(uint2); }
};

// a CTA's steps, the last of each symbol with its C
__device__ __forceinline__ const uint2* fm_load(const FmTree& t, uint2* s_steps) {
  for (uint32_t c = threadIdx.x; c < t.sigma; c += blockDim.x) {
    const uint32_t base = (uint32_t)__ldg(t.C + c), at = c * t.L;
    for (int l = 0; l < t.L; ++l) {
      uint2 v = __ldg(t.steps + at + l);
      if (l + 1 == t.L) v = make_uint2(v.x + base, v.y + base);
      s_steps[at + l] = v;
    }
  }
  __syncthreads();
  return s_steps;
}

// the rows [x, y) prefixed by pattern symbols [a, i), from the interval [x, y)
template <bool BLOCKS, bool SHARE>
__device__ __forceinline__ uint32_t fm_search(const FmTree& t, const uint2* __restrict__ st, PatternReader& rd,
                                              uint64_t a, uint64_t i, uint32_t x, uint32_t y) {
  bool known = true;  // every symbol read so far is one of the tree's
  while (known && i > a && x < y) {
    const uint32_t c = rd.at(--i);
    known = c < t.sigma;
    if (known) t.template step<BLOCKS, SHARE>(st, c, x, y);
  }
  return known && y > x ? y - x : 0;
}

// A batch that is not prepared.  Bound by the chain of its reads, which the
// compiler issues ahead where it has 48 registers (5 CTAs an SM): 2^14 patterns of
// 100 symbols, 2^24 symbols of 4 letters, 81 us, without the bound (40 registers)
// 117, at 32, which spill, 143.
__global__ void __launch_bounds__(256, 5)
    fm_count_kernel(FmTree t, const uint8_t* __restrict__ pat, const uint64_t* __restrict__ off, uint64_t m,
                    uint64_t* __restrict__ out) {
  extern __shared__ uint2 s_steps[];
  const uint2* const st = fm_load(t, s_steps);
  const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m) return;
  PatternReader rd(pat, off[m]);
  out[p] = fm_search<false, false>(t, st, rd, off[p], off[p + 1], 0u, (uint32_t)t.n);
}

// Bound by the random reads of the tree: 2^24 patterns of 8 to 32 symbols over
// a 2^28-symbol BWT of 6 symbols (3 levels, 134 MB of blocks, a third of the
// reads from L2) take 6.3 ms: 11.7 with rank entry and word apart and every
// symbol stepped, 9.9 with the interval table and shared reads, 8.3 with
// blocks, 7.1 by length, 6.3 with the blocks kept out of L1.  At 6 CTAs an SM
// (40 registers) 7.2 ms, at 8 (spills) 9.8 before that last change.
// patterns off[0..m] (total: the bytes of the whole batch) in the order of their
// lengths, so that the lanes of a warp finish together
__global__ void __launch_bounds__(256, 6)
    fm_planned_kernel(FmTree t, FmTable table, const uint8_t* __restrict__ pat, const uint64_t* __restrict__ off,
                      const uint64_t* __restrict__ total, QueryOrder ord, uint64_t m, uint64_t* __restrict__ out) {
  extern __shared__ uint2 s_steps[];
  const uint2* const st = fm_load(t, s_steps);
  uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m) return;
  const int K = table.first ? (int)ord.flags[TABLE_SYMBOLS] : 0;
  const bool blocks = t.blocks && ord.flags[MAKE_BLOCKS];
  if (!ordered_query(ord, m, p)) return;
  const uint64_t a = off[p], b = off[p + 1];
  PatternReader rd(pat, *total);
  uint32_t x = 0, y = (uint32_t)t.n;
  uint64_t i = b;
  if (K && b >= a + K) {  // (offsets that decrease: an empty pattern)
    uint32_t at = 0, scale = 1;
    bool known = true;
    for (int k = 0; k < K; ++k) {
      const uint32_t c = rd.at(--i);
      known = known && c < t.sigma;
      at += c * scale;
      scale *= (uint32_t)t.sigma;
    }
    const uint2 v = known ? __ldg(table.of(K) + at) : make_uint2(0u, 0u);
    x = v.x;
    y = v.y;
  }
  out[p] = blocks ? fm_search<true, true>(t, st, rd, a, i, x, y) : fm_search<false, true>(t, st, rd, a, i, x, y);
}

}  // namespace

int launch_fm_count(TreeImpl& t, const uint64_t* C, uint64_t sigma, const uint8_t* pat, const uint64_t* off,
                    uint64_t npat, uint64_t* out, cudaStream_t s) {
  if (!(t.flags & WTG_RANK)) return fail(WTG_ERR_INVALID, "tree built without rank support");
  if (sigma == 0 || sigma > 256 || (t.levels < 63 && sigma > (1ull << t.levels)))
    return fail(WTG_ERR_INVALID, "sigma must be 1..256 and at most 2^levels");
  if (npat == 0) return WTG_OK;
  const uint64_t* const bits = t.bits.as<uint64_t>();
  const uint64_t* const rt = t.bv.rank.as<uint64_t>();
  const Made steps(t.fm_steps, s, t.stream, true, [&](DevBuf* buf) -> int {
    const uint64_t symbols = t.levels < 8 ? 1ull << t.levels : 256;
    if (const int rc = buf[0].ensure(symbols * t.levels * sizeof(uint2), s)) return rc;
    fm_steps_kernel<<<(unsigned)((symbols + 127) / 128), 128, 0, s>>>(bits, rt, t.n, t.levels, symbols,
                                                                      buf[0].as<uint2>());
    count_launch();
    WTG_CK(cudaGetLastError());
    return WTG_OK;
  });
  if (steps.rc) return steps.rc;
  FmTree v{bits, rt, nullptr, steps.table<uint2>(0), C, t.n, sigma, t.levels};
  auto plain = [&]() -> int {
    fm_count_kernel<<<(unsigned)((npat + 255) / 256), 256, v.shared_bytes(), s>>>(v, pat, off, npat, out);
    count_launch();
    WTG_CK(cudaGetLastError());
    return WTG_OK;
  };
  if (!fm_batch_pays(npat, t.levels)) return plain();
  const uint64_t size = t.n * (uint64_t)t.levels;
  return counted_batches(
      v, off, npat, 2 * t.levels, blocks_in_reach(size), t.err, t.stream, s,
      [&](uint4* blocks, const uint32_t* wanted) { return fill_blocks(blocks, bits, rt, size, wanted, s); },
      [&](const QueryOrder& o, const FmTable& table, const uint4* blocks, uint64_t at, uint64_t m) -> int {
        v.blocks = blocks;
        fm_planned_kernel<<<(unsigned)((m + 255) / 256), 256, v.shared_bytes(), s>>>(v, table, pat, off + at, off + npat, o,
                                                                                     m, out + at);
        count_launch();
        WTG_CK(cudaGetLastError());
        return WTG_OK;
      },
      plain);
}

}  // namespace wtg
