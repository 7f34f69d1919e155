// wtg_query.cu -- batched queries on the GPU: rank_support_v::rank,
// select_support_mcl::select, and wt_int's access / rank / inverse_select /
// select, one thread per query; plus the alphabet remap helper.
#include <algorithm>

#include "wtg_blocks.cuh"
#include "wtg_order.cuh"
#include "wtg_select.cuh"
#include "wtg_tree.cuh"

namespace wtg {

__device__ __forceinline__ int bit_at(const uint64_t* __restrict__ w, uint64_t p) {
  return (int)((w[p >> 6] >> (p & 63)) & 1);
}

// Node tables: for every heap node h of levels 0..L-1 (root 0, children
// 2h+1 / 2h+2)
//   tab  : x = global bit offset of the node's start, y = ones before it --
//          the `offset` and `o = m_tree_rank(offset)` that wt_int's queries
//          recompute at every level (wt_int_par.hpp:527-536, 561-572,
//          596-606);
//   step : the two constants that take a position of the node to its child:
//          with x the position inside the level and R the ones before it
//          (rank1 of the concatenated bits), bit 0 goes on at step.x + x - R
//          and bit 1 at step.y + R, positions inside the next level; after
//          the last level the position inside the leaf.  All modulo 2^32.
//          Node h at step[h + 1], so that the children lie in one 16 bytes.
// With step, a query level costs one rank entry, one word and 8 bytes of a
// table that is read beside them; tab took two 16-byte entries a level.
__global__ void node_table_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt,
                                  const uint32_t* __restrict__ Z, const uint32_t* __restrict__ C, uint64_t n, int L,
                                  uint64_t nodes, ulonglong2* __restrict__ tab, uint2* __restrict__ step) {
  const uint64_t h = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= nodes) return;
  const uint64_t l = 63 - __clzll((long long)(h + 1));
  const uint32_t c = C[h];
  const uint64_t off = l * n + c;
  const uint64_t y = rank1_dev(rt, tree, off);
  tab[h] = make_ulonglong2(off, y);
  const uint32_t Y = (uint32_t)y;
  step[h + 1] = (int)l + 1 < L ? make_uint2(Y, c + Z[h] - Y) : make_uint2(Y - c, 0u - Y);
}

// What the descents probe: the rank table and the bitvector, or for large
// sorted batches the blocks made of them (one sector a level instead of two:
// the sorted descent is bound by the lines its loads look up in L1).
template <bool BLOCKS>
struct LevelBits {
  const uint64_t* tree;
  const uint64_t* rt;
  const uint4* blocks;
  // ones before pos (mod 2^32), and the bit at it
  __device__ __forceinline__ uint32_t rank(uint64_t pos, uint32_t& bit) const {
    if constexpr (BLOCKS) {
      uint32_t off;
      uint64_t v[4];
      block_load(blocks, block_of(pos, off), v);
      const BlockProbe r = block_at(v, off);
      bit = r.bit;
      return r.ones;
    } else {
      const ulonglong2 e = load_entry(rt, pos);
      const uint64_t word = load_word(tree, pos);
      bit = (uint32_t)(word >> (pos & 63)) & 1u;
      return entry_rank(e, word, pos);
    }
  }
};

// wt_int::operator[] (wt_int/wt_int_par.hpp:519-541) and inverse_select
// (:588-611): descend by the bit at i; the symbol is the path, the rank the
// final position
template <bool INV, bool BLOCKS>
__device__ __forceinline__ void descend(const LevelBits<BLOCKS>& bits, const uint2* __restrict__ step, uint64_t n, int L,
                                        uint64_t i, uint64_t k, uint64_t* __restrict__ out,
                                        uint64_t* __restrict__ sym_out) {
  uint32_t x = (uint32_t)i, h = 1;  // h: heap id + 1, the path with a leading 1
  uint64_t lbase = 0;
  uint2 st = __ldg(step + 1);
  for (int lv = 0; lv < L; ++lv, lbase += n) {
    // the children's constants come with this level's reads, not after them
    uint4 next = make_uint4(0u, 0u, 0u, 0u);
    if (lv + 1 < L) next = __ldg(reinterpret_cast<const uint4*>(step + 2 * h));
    uint32_t bit;
    const uint32_t R = bits.rank(lbase + x, bit);
    x = bit ? st.y + R : st.x + x - R;
    st = bit ? make_uint2(next.z, next.w) : make_uint2(next.x, next.y);
    h = 2 * h + bit;
  }
  const uint64_t c = h - (1u << L);
  if (INV) {
    out[k] = x;
    sym_out[k] = c;
  } else {
    out[k] = c;
  }
}

// A batch that came in order (see order_check_kernel) is read as it is, without
// the blocks, which were not made for it.
template <bool INV, bool ORD, bool BLOCKS>
__global__ void wt_descend_kernel(LevelBits<BLOCKS> bits, const uint2* __restrict__ step, uint64_t n, int L,
                                  const uint64_t* __restrict__ q, QueryOrder ord, uint64_t nq,
                                  uint64_t* __restrict__ out, uint64_t* __restrict__ sym_out) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  const bool as_is = !ORD || ord.flags[AS_IS];
  const uint64_t i = as_is ? q[k] : ord.pos[k];
  if (ORD && !ordered_query(ord, nq, k)) return;
  if (i >= n) {
    out[k] = NONE64;
    if (INV) sym_out[k] = NONE64;
    return;
  }
  if (BLOCKS && as_is) descend<INV>(LevelBits<false>{bits.tree, bits.rt, nullptr}, step, n, L, i, k, out, sym_out);
  else descend<INV>(bits, step, n, L, i, k, out, sym_out);
}

// wt_int::rank (wt_int_par.hpp:553-577): descend along c's path
template <bool BLOCKS>
__device__ __forceinline__ uint32_t rank_along(const LevelBits<BLOCKS>& bits, const uint2* __restrict__ step, uint64_t n,
                                               int L, uint32_t x, uint32_t c) {
  const uint32_t path = c | (1u << L);
  uint64_t lbase = 0;
  uint2 st = __ldg(step + 1);
  for (int lv = 0; lv < L; ++lv, lbase += n) {
    const uint2 next = __ldg(step + (path >> (lv + 1 < L ? L - 1 - lv : L)));  // one level ahead
    uint32_t bit;
    const uint32_t R = bits.rank(lbase + x, bit);
    x = (path >> (L - 1 - lv)) & 1u ? st.y + R : st.x + x - R;
    st = next;
  }
  return x;
}

// the same by node entries (see the far kernels).  (The test of the offset is
// the compiler's better code: 2^22 consecutive positions, 2^28 symbols x 20
// levels 363 us, without it 391.)
__device__ __forceinline__ uint64_t rank_far(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt,
                                             const ulonglong2* __restrict__ tab, int L, uint64_t i, uint64_t c) {
  uint64_t h = 0;
  ulonglong2 nd = __ldg(tab);
  for (int lv = 0; lv < L && i; ++lv) {
    const uint64_t bit = (c >> (L - 1 - lv)) & 1;
    const uint64_t child = 2 * h + 1 + bit;
    ulonglong2 next = nd;
    if (lv + 1 < L) next = __ldg(tab + child);
    const uint64_t pos = nd.x + i;
    const uint64_t word = load_word(tree, pos);
    const ulonglong2 e = load_entry(rt, pos);
    uint64_t r = e.x + ((e.y >> (63 - 9 * ((pos & 0x1FF) >> 6))) & 0x1FF);
    if (pos & 63) r += __popcll(word & ((1ull << (pos & 63)) - 1));
    r -= nd.y;
    i = bit ? r : i - r;
    h = child;
    nd = next;
  }
  return i;
}

// far: a batch that came in order goes by node entries (see launch_wt_rank)
template <bool ORD, bool BLOCKS>
__global__ void wt_rank_kernel(LevelBits<BLOCKS> bits, const uint2* __restrict__ step,
                               const ulonglong2* __restrict__ tab, uint64_t n, int L, const uint64_t* __restrict__ q,
                               QueryOrder ord, bool far, const uint64_t* __restrict__ sym, uint64_t nq,
                               uint64_t* __restrict__ out) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  if (ORD && !ordered_query(ord, nq, k)) return;
  const uint64_t i = q[k];
  const uint64_t c = sym[k];
  if (i > n) {
    out[k] = NONE64;
    return;
  }
  if (L < 64 && (1ull << L) <= c) {
    out[k] = 0;
    return;
  }
  const bool as_is = ORD && ord.flags[AS_IS];
  if (as_is && far) out[k] = rank_far(bits.tree, bits.rt, tab, L, i, c);
  else if (as_is)
    out[k] = rank_along(LevelBits<false>{bits.tree, bits.rt, nullptr}, step, n, L, (uint32_t)i, (uint32_t)c);
  else out[k] = rank_along(bits, step, n, L, (uint32_t)i, (uint32_t)c);
}

// Descents of batches that are not sorted, over trees larger than L2: node
// entries and positions inside the node, 64-bit.  They read the same lines as
// the kernels above and are slower by 10 % where L2 holds the tree, but their
// queries stay together level by level (the levels of all queries in flight
// must meet in L2: 0.72 GB from DRAM where the other rank read 1.01 GB, at 80 %
// of its bandwidth both): 2^28 x 12 levels, rank of 2^19 queries 0.11 ms
// against 0.15, access of 2^18 66 us against 70.
__device__ __forceinline__ uint64_t entry_rank64(const ulonglong2& e, uint64_t word, uint64_t pos) {
  return e.x + ((e.y >> (63 - 9 * ((pos >> 6) & 7))) & 0x1FF) + __popcll(word & ((1ull << (pos & 63)) - 1));
}

template <bool INV>
__global__ void wt_descend_far_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt,
                                  const ulonglong2* __restrict__ tab, uint64_t n, int L,
                                  const uint64_t* __restrict__ q, uint64_t nq, uint64_t* __restrict__ out,
                                  uint64_t* __restrict__ sym_out) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  uint64_t i = q[k];
  if (i >= n) {
    out[k] = NONE64;
    if (INV) sym_out[k] = NONE64;
    return;
  }
  uint64_t h = 0, c = 0;
  ulonglong2 nd = __ldg(tab);
  for (int lv = 0; lv < L; ++lv) {
    const uint64_t pos = nd.x + i;
    ulonglong2 c0 = nd, c1 = nd;
    if (lv + 1 < L) {
      c0 = __ldg(tab + 2 * h + 1);
      c1 = __ldg(tab + 2 * h + 2);
    }
    const uint64_t word = load_word(tree, pos);
    const uint64_t r = entry_rank64(load_entry(rt, pos), word, pos) - nd.y;
    const uint64_t bit = (word >> (pos & 63)) & 1;
    c = (c << 1) | bit;
    if (bit) {
      i = r;
      h = 2 * h + 2;
      nd = c1;
    } else {
      i -= r;
      h = 2 * h + 1;
      nd = c0;
    }
  }
  if (INV) {
    out[k] = i;
    sym_out[k] = c;
  } else {
    out[k] = c;
  }
}

__global__ void wt_rank_far_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt,
                                   const ulonglong2* __restrict__ tab, uint64_t n, int L,
                                   const uint64_t* __restrict__ q, const uint64_t* __restrict__ sym, uint64_t nq,
                                   uint64_t* __restrict__ out) {
  const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  const uint64_t i = q[k];
  const uint64_t c = sym[k];
  if (i > n) {
    out[k] = NONE64;
    return;
  }
  if (L < 64 && (1ull << L) <= c) {
    out[k] = 0;
    return;
  }
  out[k] = rank_far(tree, rt, tab, L, i, c);
}

// wt_int::select (wt_int_par.hpp:622-660): down c's path for the nodes' starts
// and the ones before them, then up by the selects.  TAB: starts and ones are
// the node table's and the occurrences of c a leaf's size, so that nothing but
// the selects waits for one another (a call of 1000 over 2^20 x 8 levels 73 / 70
// us, over 2^22 x 20 108 / 95, of 2^18 293 / 255).
template <bool TAB, bool WORDS>
__global__ void wt_select_kernel(const uint64_t* __restrict__ tree, const uint64_t* __restrict__ rt, SelView s1,
                                 SelView s0, const ulonglong2* __restrict__ tab, const uint32_t* __restrict__ C, uint64_t n,
                                 int L, const uint64_t* __restrict__ q,
                                 const uint64_t* __restrict__ sym, uint64_t nq, uint64_t* __restrict__ out) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  uint64_t i = q[k];
  const uint64_t c = sym[k];
  if (i == 0 || (L < 64 && (1ull << L) <= c)) {
    out[k] = NONE64;
    return;
  }
  if constexpr (TAB) {
    const uint32_t path = (uint32_t)c | (1u << L);  // path >> (L - l): heap id + 1 of level l's node
    const uint32_t last = path >> 1;                // of the last level's
    ulonglong2 nd = __ldg(tab + (last - 1));
    const uint32_t from = __ldg(C + (last - 1));
    const uint64_t to = last & (last + 1) ? __ldg(C + last) : (uint32_t)n;  // the level's last node ends at n
    const uint64_t ones = rank1_dev(rt, tree, nd.x + (to - from)) - nd.y;
    const uint64_t occ = path & 1u ? ones : to - from - ones;
    if (occ < i) {
      out[k] = NONE64;  // the reference throws std::logic_error here
      return;
    }
    for (int lv = L; lv > 0; --lv) {
      const ulonglong2 up = __ldg(tab + (lv > 1 ? (path >> (L - lv + 2)) - 1 : 0));
      if ((path >> (L - lv)) & 1u) i = select_dev<WORDS>(s1, nd.y + i) - nd.x + 1;
      else i = select_dev<WORDS>(s0, nd.x - nd.y + i) - nd.x + 1;
      nd = up;
    }
    out[k] = i - 1;
    return;
  }
  uint64_t path_off[25], path_rank[25];
  uint64_t offset = 0, mask = 1ull << (L - 1), node_size = n;
  path_off[0] = path_rank[0] = 0;
  for (int lv = 0; lv < L && node_size; ++lv) {
    const uint64_t o = rank1_dev(rt, tree, offset);
    path_rank[lv] = o;
    const uint64_t oe = rank1_dev(rt, tree, offset + node_size) - o;
    if (c & mask) {
      offset += node_size - oe;
      node_size = oe;
    } else {
      node_size = node_size - oe;
    }
    offset += n;
    path_off[lv + 1] = offset;
    mask >>= 1;
  }
  if (node_size == 0 || node_size < i) {
    out[k] = NONE64;  // the reference throws std::logic_error here
    return;
  }
  mask = 1;
  for (int lv = L; lv > 0; --lv) {
    offset = path_off[lv - 1];
    const uint64_t o = path_rank[lv - 1];
    if (c & mask) i = select_dev<WORDS>(s1, o + i) - offset + 1;
    else i = select_dev<WORDS>(s0, offset - o + i) - offset + 1;
    mask <<= 1;
  }
  out[k] = i - 1;
}

__global__ void bv_rank_kernel(const uint64_t* __restrict__ words, const uint64_t* __restrict__ rt, uint64_t size,
                               const uint64_t* __restrict__ q, uint64_t nq, uint64_t* __restrict__ out) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  const uint64_t idx = q[k];
  out[k] = idx <= size ? rank1_dev(rt, words, idx) : NONE64;
}

template <bool WORDS>
__global__ void bv_select_kernel(SelView v, const uint64_t* __restrict__ q, uint64_t nq, uint64_t* __restrict__ out) {
  uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nq) return;
  out[k] = select_dev<WORDS>(v, q[k]);
}

static unsigned qgrid(uint64_t nq) { return (unsigned)((nq + 255) / 256); }

static int need(const TreeImpl& t, uint32_t f, const char* what) {
  if ((t.flags & f) != f) return fail(WTG_ERR_INVALID, std::string(what) + " needs a tree built with the supports it uses");
  return WTG_OK;
}

WTG_WAIT_LIMIT_SETTER(query)

static int make_node_tables(const TreeImpl& t, DevBuf* buf, cudaStream_t s) {
  int rc;
  const uint64_t heap = 1ull << t.levels, nodes = heap - 1;
  if ((rc = buf[0].ensure(nodes * sizeof(ulonglong2), s))) return rc;
  if ((rc = buf[1].ensure((nodes + 1) * sizeof(uint2), s))) return rc;
  node_table_kernel<<<(unsigned)((nodes + 255) / 256), 256, 0, s>>>(
      t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), t.zeros.as<uint32_t>(), t.zeros.as<uint32_t>() + heap, t.n,
      t.levels, nodes, buf[0].as<ulonglong2>(), buf[1].as<uint2>());
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

NodeTables::NodeTables(TreeImpl& t, cudaStream_t s, bool make)
    : Made(t.node_tables, s, t.stream, make, [&](DevBuf* buf) { return make_node_tables(t, buf, s); }),
      tab(table<ulonglong2>(0)), step(table<uint2>(1)) {}

// Blocks (built from the bitvector for the call: 1.1 ms for 2^30 x 20 levels,
// 112 M blocks) pay once the batch probes a good part of them and there are
// levels enough.  Access, sorted, ms without / with blocks: 2^30 x 20, 2^26
// queries 14.2 / 11.3, 2^25 7.00 / 6.07, 2^24 3.42 / 3.39, 2^23 1.63 / 2.10;
// 2^27 x 20 (14 M blocks), 2^26 6.52 / 5.98, 2^23 0.89 / 0.86, 2^22 0.48 /
// 0.53; but 2^28 x 8 (11 M), 2^26 4.52 / 4.28, 2^25 2.19 / 2.17, 2^24 1.04 / 1.10.
static bool blocks_pay(const TreeImpl& t, uint64_t nq) {
  return order_pays(t, nq, false) && t.levels >= 12 && nq >= block_count(t.n * (uint64_t)t.levels) / 3;
}

// (below 2^17 queries the tree's lines that they read stay in L2)
static bool far_descent(const TreeImpl& t, uint64_t nq) { return larger_than_l2(t) && nq >= (1ull << 17); }

// in_order, with the blocks where they pay and there is room for them:
// launch(nodes, bits, ordered, order, first query, queries), ordered a bool constant
template <typename F>
static int descents(TreeImpl& t, const uint64_t* idx, uint64_t nq, cudaStream_t s, F launch) {
  if (!nq) return WTG_OK;
  const NodeTables nodes(t, s);
  if (nodes.rc) return nodes.rc;
  const uint64_t* const words = t.bits.as<uint64_t>();
  const uint64_t* const rt = t.bv.rank.as<uint64_t>();
  uint4* blocks = nullptr;
  const int rc = in_order(t, false, idx, nq, s, [&](bool sorted, const QueryOrder& o, uint64_t at, uint64_t m) -> int {
    if (sorted && blocks_pay(t, nq)) {
      // (once the sort has its scratch, which comes first; by the first batch that does not come in order)
      const uint64_t size = t.n * (uint64_t)t.levels;
      if (!at) blocks = (uint4*)try_scratch(block_count(size) * 32, s);
      if (blocks && !fill_blocks(blocks, words, rt, size, o.flags + MAKE_BLOCKS, s))
        return fail(WTG_ERR_CUDA, "query blocks: launch failed");
    }
    if (sorted && blocks) launch(nodes, LevelBits<true>{words, rt, blocks}, std::true_type{}, o, at, m);
    else if (sorted) launch(nodes, LevelBits<false>{words, rt, nullptr}, std::true_type{}, o, at, m);
    else launch(nodes, LevelBits<false>{words, rt, nullptr}, std::false_type{}, o, at, m);
    count_launch();
    WTG_CK(cudaGetLastError());
    return WTG_OK;
  });
  if (blocks) cudaFreeAsync(blocks, s);
  return rc;
}

int launch_wt_access(TreeImpl& t, const uint64_t* idx, uint64_t nq, uint64_t* out, cudaStream_t s) {
  if (int rc = need(t, WTG_RANK, "access")) return rc;
  return descents(t, idx, nq, s, [&](const NodeTables& nodes, auto bits, auto ord, const QueryOrder& o, uint64_t at,
                                     uint64_t m) {
    if (!ord() && far_descent(t, m))
      wt_descend_far_kernel<false><<<qgrid(m), 256, 0, s>>>(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), nodes.tab,
                                                            t.n, t.levels, idx + at, m, out + at, nullptr);
    else
      wt_descend_kernel<false, ord()><<<qgrid(m), 256, 0, s>>>(bits, nodes.step, t.n, t.levels, idx + at, o, m,
                                                               out + at, nullptr);
  });
}

int launch_wt_rank(TreeImpl& t, const uint64_t* idx, const uint64_t* sym, uint64_t nq, uint64_t* out,
                   cudaStream_t s) {
  if (int rc = need(t, WTG_RANK, "rank")) return rc;
  // 2^22 consecutive positions, us by steps / by node entries: 2^28 symbols x 8
  // levels 99 / 110, x 12 118 / 135, x 20 385 / 363, 2^29 x 20 503 / 419
  const bool far = t.levels >= 16;
  return descents(t, idx, nq, s, [&](const NodeTables& nodes, auto bits, auto ord, const QueryOrder& o, uint64_t at,
                                     uint64_t m) {
    if (!ord() && far_descent(t, m))
      wt_rank_far_kernel<<<qgrid(m), 256, 0, s>>>(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), nodes.tab, t.n,
                                                  t.levels, idx + at, sym + at, m, out + at);
    else
      wt_rank_kernel<ord()><<<qgrid(m), 256, 0, s>>>(bits, nodes.step, nodes.tab, t.n, t.levels, idx + at, o, far,
                                                     sym + at, m, out + at);
  });
}

int launch_wt_inverse_select(TreeImpl& t, const uint64_t* idx, uint64_t nq, uint64_t* rank_out,
                             uint64_t* sym_out, cudaStream_t s) {
  if (int rc = need(t, WTG_RANK, "inverse_select")) return rc;
  return descents(t, idx, nq, s, [&](const NodeTables& nodes, auto bits, auto ord, const QueryOrder& o, uint64_t at,
                                     uint64_t m) {
    if (!ord() && far_descent(t, m))
      wt_descend_far_kernel<true><<<qgrid(m), 256, 0, s>>>(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), nodes.tab,
                                                           t.n, t.levels, idx + at, m, rank_out + at, sym_out + at);
    else
      wt_descend_kernel<true, ord()><<<qgrid(m), 256, 0, s>>>(bits, nodes.step, t.n, t.levels, idx + at, o, m,
                                                              rank_out + at, sym_out + at);
  });
}

int launch_wt_select(TreeImpl& t, const uint64_t* i, const uint64_t* sym, uint64_t nq, uint64_t* out,
                     cudaStream_t s) {
  if (int rc = need(t, WTG_ALL, "select")) return rc;
  if (!nq) return WTG_OK;
  // the node table where there is one, or the batch is worth making it (24
  // bytes and a rank per node) and there is room
  const uint64_t heap = 1ull << t.levels;
  const NodeTables nodes(t, s, heap <= 8 * nq);
  if (nodes.rc) cudaGetLastError();
  const bool tab = t.n && nodes.rc == WTG_OK && nodes.tab;
  // a call of 2^16 queries, us word by word / by sectors: 2^28 symbols x 20 levels 194
  // / 172, x 8 116 / 105; 2^18: 283 / 358, 182 / 220, 2^22 x 20 248 / 282
  const bool many = nq >= SEL_MANY;
  auto* const f = many ? tab ? wt_select_kernel<true, true> : wt_select_kernel<false, true>
                       : tab ? wt_select_kernel<true, false> : wt_select_kernel<false, false>;
  f<<<qgrid(nq), 256, 0, s>>>(t.bits.as<uint64_t>(), t.bv.rank.as<uint64_t>(), sel_view(t.bv, 1), sel_view(t.bv, 0),
                              nodes.tab, t.zeros.as<uint32_t>() + heap, t.n, t.levels, i, sym, nq, out);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

int launch_bv_rank(const BvSupport& bv, const uint64_t* idx, uint64_t nq, uint64_t* out, cudaStream_t s) {
  if (!(bv.flags & WTG_RANK)) return fail(WTG_ERR_INVALID, "rank needs WTG_RANK");
  if (!nq) return WTG_OK;
  bv_rank_kernel<<<qgrid(nq), 256, 0, s>>>(bv.words, bv.rank.as<uint64_t>(), bv.size, idx, nq, out);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

int launch_bv_select(const BvSupport& bv, int t_b, const uint64_t* i, uint64_t nq, uint64_t* out, cudaStream_t s) {
  if (!(bv.flags & (t_b ? WTG_SELECT1 : WTG_SELECT0))) return fail(WTG_ERR_INVALID, "select needs its support built");
  if (!nq) return WTG_OK;
  auto* const f = select_by_words(bv.sel[t_b], bv.size, nq) ? bv_select_kernel<true> : bv_select_kernel<false>;
  f<<<qgrid(nq), 256, 0, s>>>(sel_view(bv, t_b), i, nq, out);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

// ---------------------------------------------------------- alphabet remap

template <typename T>
__global__ void remap_mark_kernel(const T* __restrict__ s, uint64_t n, uint32_t* __restrict__ flag) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    flag[(uint64_t)s[i]] = 1;
}

template <typename T>
__global__ void remap_apply_kernel(T* __restrict__ s, uint64_t n, const uint32_t* __restrict__ rank) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    s[i] = (T)rank[(uint64_t)s[i]];
}

template <typename T>
__global__ void remap_max_kernel(const T* __restrict__ s, uint64_t n, unsigned long long* out) {
  uint64_t m = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t x = s[i];
    m = x > m ? x : m;
  }
  atomicMax(out, (unsigned long long)m);
}

template <typename T>
static int remap_t(T* d, uint64_t n, uint64_t* sigma, DevBuf& tmp, DevBuf& scan_tmp, uint32_t* d_err,
                   cudaStream_t s) {
  int rc;
  unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, 152 * 8);
  if (grid == 0) grid = 1;
  if ((rc = tmp.ensure(sizeof(unsigned long long), s))) return rc;
  WTG_CK(cudaMemsetAsync(tmp.p, 0, sizeof(unsigned long long), s));
  remap_max_kernel<T><<<grid, 256, 0, s>>>(d, n, tmp.as<unsigned long long>());
  count_launch();
  WTG_CK(cudaGetLastError());
  unsigned long long mx = 0;
  WTG_CK(cudaMemcpyAsync(&mx, tmp.p, sizeof(mx), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));
  if (mx >= (1ull << 31)) return fail(WTG_ERR_RANGE, "remap: symbol values must be below 2^31");
  const uint64_t k = mx + 2;  // flags for values 0..max, plus the total
  if ((rc = tmp.ensure(k * sizeof(uint32_t), s))) return rc;
  uint32_t* flag = tmp.as<uint32_t>();
  WTG_CK(cudaMemsetAsync(flag, 0, k * sizeof(uint32_t), s));
  remap_mark_kernel<T><<<grid, 256, 0, s>>>(d, n, flag);
  count_launch();
  WTG_CK(cudaGetLastError());
  if ((rc = scan_exclusive_u32(flag, flag, k, scan_tmp, d_err, s))) return rc;
  remap_apply_kernel<T><<<grid, 256, 0, s>>>(d, n, flag);
  count_launch();
  WTG_CK(cudaGetLastError());
  uint32_t sg = 0;
  WTG_CK(cudaMemcpyAsync(&sg, flag + (k - 1), sizeof(sg), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));
  *sigma = sg;
  return WTG_OK;
}

int remap_alphabet_device(void* d_seq, uint64_t n, int eb, uint64_t* sigma, DevBuf& tmp, DevBuf& scan_tmp,
                          uint32_t* d_err, cudaStream_t s) {
  if (n == 0) {
    *sigma = 0;
    return WTG_OK;
  }
  switch (eb) {
    case 1: return remap_t<uint8_t>((uint8_t*)d_seq, n, sigma, tmp, scan_tmp, d_err, s);
    case 2: return remap_t<uint16_t>((uint16_t*)d_seq, n, sigma, tmp, scan_tmp, d_err, s);
    case 4: return remap_t<uint32_t>((uint32_t*)d_seq, n, sigma, tmp, scan_tmp, d_err, s);
    default: return remap_t<uint64_t>((uint64_t*)d_seq, n, sigma, tmp, scan_tmp, d_err, s);
  }
}

}  // namespace wtg
