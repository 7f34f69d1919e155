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
// each symbol's step constants are tabulated once per call (fm_steps_kernel; in
// scratch of the call, as they hold its C) and kept in shared memory; a rank
// then costs one rank_support_v probe per level, and sp and ep share the path
// -- and, once the interval is short, the rank entry and the word.  The last K symbols of a pattern come from a table
// of the intervals of all strings of K symbols, made once per call where the
// batch is much larger than the table (wtg_fm_table.cuh).
#include "wtg_blocks.cuh"
#include "wtg_fm_table.cuh"
#include "wtg_order.cuh"
#include "wtg_select.cuh"
#include "wtg_tree.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(fm)

namespace {

constexpr int FM_SMEM_STEPS = 2048;  // steps kept in shared memory (8 bytes each)

// steps[c * L + l]: with x a position of c's node inside level l and R the
// ones before it, bit 0 of c's path goes on at .x + x - R, bit 1 at .y + R
// (mod 2^32; see node_table_kernel); after the last level the result is
// C[c] + rank(., c)
__global__ void fm_steps_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt, uint64_t n, int L,
                                uint64_t sigma, const uint64_t* __restrict__ C, uint2* __restrict__ steps) {
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= sigma) return;
  uint64_t offset = 0, size = n;
  for (int l = 0; l < L; ++l) {
    const uint64_t o = rank1_dev(rt, tree, offset);
    const uint64_t oe = rank1_dev(rt, tree, offset + size) - o;
    const uint32_t Y = (uint32_t)o, start = (uint32_t)(offset - (uint64_t)l * n);
    const uint32_t zeros = (uint32_t)(size - oe);
    if (l + 1 < L) steps[c * L + l] = make_uint2(Y, start + zeros - Y);
    else steps[c * L + l] = make_uint2((uint32_t)C[c] + Y - start, (uint32_t)C[c] - Y);
    if ((c >> (L - 1 - l)) & 1) {
      offset += size - oe;
      size = oe;
    } else {
      size -= oe;
    }
    offset += n;
  }
}

// the tree with its rank table (BLOCKS false) or as 192-bit blocks
template <bool BLOCKS>
struct FmTree {
  const uint64_t* tree;
  const uint64_t* rt;
  const uint4* blocks;
  const uint2* steps;
  uint64_t n, sigma;
  int L;
  // ones before the positions px <= py.  SHARE: what they share is read once,
  // for batches bound by their reads; a small batch waits for its reads, and
  // the second would wait for the first (2^14 patterns: 58 us against 67)
  template <bool SHARE>
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
  // prepends symbol c (< sigma) to the interval [x, y)
  template <bool SHARE>
  __device__ __forceinline__ void step(const uint2* __restrict__ st, uint32_t c, uint32_t& x, uint32_t& y) const {
    uint64_t lbase = 0;
    for (int l = 0; l < L; ++l, lbase += n) {
      const uint2 s = st[c * L + l];
      uint32_t rx, ry;
      ranks<SHARE>(lbase + x, lbase + y, rx, ry);
      const bool one = (c >> (L - 1 - l)) & 1;
      x = one ? s.y + rx : s.x + x - rx;
      y = one ? s.y + ry : s.x + y - ry;
    }
  }
};

// intervals of all strings of k symbols from those of k - 1 (k = 1: from the
// whole range): string c w at c sigma^(k-1) + w
template <bool BLOCKS>
__global__ void fm_table_kernel(FmTree<BLOCKS> t, uint64_t prev_count, const uint2* __restrict__ prev,
                                uint2* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= prev_count * t.sigma) return;
  const uint32_t c = (uint32_t)(i / prev_count);
  const uint2 v = prev ? prev[i - c * prev_count] : make_uint2(0u, (uint32_t)t.n);
  uint32_t x = v.x, y = v.y;
  if (x < y) t.template step<true>(t.steps, c, x, y);
  out[i] = x < y ? make_uint2(x, y) : make_uint2(0u, 0u);
}

// Bound by the random reads of the tree: 2^24 patterns of 8 to 32 symbols over
// a 2^28-symbol BWT of 6 symbols (3 levels, 134 MB of blocks, a third of the
// reads from L2) take 6.3 ms: 11.7 with rank entry and word apart and every
// symbol stepped, 9.9 with the interval table and shared reads, 8.3 with
// blocks, 7.1 by length, 6.3 with the blocks kept out of L1.  At 6 CTAs an SM
// (40 registers) 7.2 ms, at 8 (spills) 9.8 before that last change.
// ORD: patterns off[0..m] (total: the bytes of the whole batch) in the order
// of their lengths, so that the lanes of a warp finish together
template <bool BLOCKS, bool ORD>
__global__ void __launch_bounds__(256, 6)
    fm_count_kernel(FmTree<BLOCKS> t, int K, const uint2* __restrict__ table, const uint8_t* __restrict__ pat,
                    const uint64_t* __restrict__ off, const uint64_t* __restrict__ total, QueryOrder ord, uint64_t m,
                    uint64_t* __restrict__ out) {
  __shared__ uint2 s_steps[FM_SMEM_STEPS];
  const uint32_t nsteps = (uint32_t)t.sigma * t.L;
  const bool in_smem = nsteps <= (uint32_t)FM_SMEM_STEPS;
  if (in_smem)
    for (uint32_t i = threadIdx.x; i < nsteps; i += blockDim.x) s_steps[i] = t.steps[i];
  __syncthreads();
  const uint2* const st = in_smem ? s_steps : t.steps;
  uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= m) return;
  if (ORD && !ordered_query(ord, m, p)) return;
  const uint64_t a = off[p], b = off[p + 1];
  PatternReader rd(pat, *total);
  uint32_t x = 0, y = (uint32_t)t.n;
  uint64_t i = b;
  bool known = true;  // every symbol read so far is one of the tree's
  if (K && b >= a + K) {  // (offsets that decrease: an empty pattern)
    uint32_t at = 0, scale = 1;
    for (int k = 0; k < K; ++k) {
      const uint32_t c = rd.at(--i);
      known = known && c < t.sigma;
      at += c * scale;
      scale *= (uint32_t)t.sigma;
    }
    if (known) {
      const uint2 v = __ldg(table + at);
      x = v.x;
      y = v.y;
    }
  }
  while (known && i > a && x < y) {
    const uint32_t c = rd.at(--i);
    known = c < t.sigma;
    if (known) t.template step<ORD>(st, c, x, y);
  }
  out[p] = known && y > x ? y - x : 0;
}

template <bool BLOCKS>
int fm_run(TreeImpl& t, const uint4* blocks, const uint2* steps, uint64_t sigma, const uint8_t* pat, const uint64_t* off, uint64_t npat,
           uint64_t* out, cudaStream_t s) {
  const FmTree<BLOCKS> v{t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), blocks, steps, t.n, sigma, t.levels};
  const bool pays = fm_batch_pays(npat, t.levels);
  return with_fm_table<uint2>(
      pays, sigma, npat, s,
      [&](uint64_t prev_count, const uint2* prev, uint2* next) -> int {
        fm_table_kernel<BLOCKS><<<(unsigned)((prev_count * sigma + 127) / 128), 128, 0, s>>>(v, prev_count, prev, next);
        count_launch();
        WTG_CK(cudaGetLastError());
        return WTG_OK;
      },
      [&](int K, const uint2* table) -> int {
        return by_length(pays, off, npat, t.err, t.stream, s,
                         [&](bool sorted, const QueryOrder& o, uint64_t at, uint64_t m) -> int {
                           auto* const f = sorted ? fm_count_kernel<BLOCKS, true> : fm_count_kernel<BLOCKS, false>;
                           f<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(v, K, table, pat, off + at, off + npat, o, m,
                                                                         out + at);
                           count_launch();
                           WTG_CK(cudaGetLastError());
                           return WTG_OK;
                         });
      });
}

}  // namespace

int launch_fm_count(TreeImpl& t, const uint64_t* C, uint64_t sigma, const uint8_t* pat, const uint64_t* off,
                    uint64_t npat, uint64_t* out, cudaStream_t s) {
  int rc;
  if (!(t.flags & WTG_RANK)) return fail(WTG_ERR_INVALID, "tree built without rank support");
  if (sigma == 0 || sigma > 256 || (t.levels < 63 && sigma > (1ull << t.levels)))
    return fail(WTG_ERR_INVALID, "sigma must be 1..256 and at most 2^levels");
  if (npat == 0) return WTG_OK;
  struct Steps : DevBuf {
    cudaStream_t s;
    explicit Steps(cudaStream_t st) : s(st) {}
    ~Steps() { release(s); }
  } steps(s);
  if ((rc = steps.ensure(sigma * t.levels * sizeof(uint2), s))) return rc;
  fm_steps_kernel<<<(unsigned)((sigma + 127) / 128), 128, 0, s>>>(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), t.n,
                                                                  t.levels, sigma, C, steps.as<uint2>());
  count_launch();
  WTG_CK(cudaGetLastError());
  // blocks pay once the batch probes a good part of them: making them is a
  // read and write of the bits (35 us for 8e8 bits), a probe saves a sector
  const uint64_t size = t.n * (uint64_t)t.levels;
  uint4* blocks = fm_batch_pays(npat, t.levels) && npat >= block_count(size) / 8
                      ? make_blocks(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), size, s)
                      : nullptr;
  rc = blocks ? fm_run<true>(t, blocks, steps.as<uint2>(), sigma, pat, off, npat, out, s)
              : fm_run<false>(t, blocks, steps.as<uint2>(), sigma, pat, off, npat, out, s);
  if (blocks) cudaFreeAsync(blocks, s);
  return rc;
}

}  // namespace wtg
