// wtg_build.cu -- level-by-level wavelet-tree construction on the GPU: the
// host side of the level passes (wtg_levels.cuh) and the node records.
//
// The reference (wavelet/levelWT/WT.C:43-227) walks the tree node by node:
// at level l every node writes bit (levels-l-1) of its symbols at
// l*n + position and stably partitions them, zeros first, into the next
// level's buffer.  Here the levels are taken in groups of up to four, each
// one count pass over the sequence, one kernel over the group's nodes and
// one pass that writes the bits of all its levels and the sequence in the
// order of the next group.  The node table (WT.C:67,113-116,191-214) follows
// from the per-node starts and left-child sizes alone.
#include <algorithm>

#include "wtg_internal.cuh"
#include "wtg_pass.cuh"
#include "wtg_tree.cuh"

namespace wtg {

template <typename T>
__global__ void max_kernel(const T* __restrict__ s, uint64_t n, unsigned long long* out) {
  uint64_t m = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    uint64_t x = s[i];
    m = x > m ? x : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    uint64_t t = __shfl_xor_sync(0xffffffffu, m, o);
    m = t > m ? t : m;
  }
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, (unsigned long long)m);
}

// Heap id h = 2^l - 1 + p names node p of level l (levelWT/WT.C:191-214).
// C[h] = start of node h in its level, Z[h] = size of its left child.

__device__ __forceinline__ void heap_split(uint64_t h, int& l, uint64_t& p) {
  l = 63 - __clzll((long long)(h + 1));
  p = h + 1 - (1ull << l);
}

// WTnode records in heap order (levelWT/WT.C:46-67,113-116,191-214).
__global__ void node_kernel(const uint32_t* __restrict__ C, const uint32_t* __restrict__ Z, int L, uint64_t n,
                            uint64_t n_entries, int ib, void* __restrict__ out) {
  uint64_t h = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n_entries) return;
  const uint64_t none = ib == 4 ? 0xFFFFFFFFull : ~0ull;
  uint64_t rec[5] = {0, 0, 0, 0, 0};
  if (h == 0) rec[2] = none;
  if (h < (1ull << L) - 1) {
    int l;
    uint64_t p;
    heap_split(h, l, p);
    const uint32_t start = C[h];
    const uint32_t len = (p + 1 < (1ull << l)) ? C[h + 1] - start : (uint32_t)n - start;
    if (h == 0 || len > 0) {
      rec[0] = (uint64_t)l * n + start;
      rec[1] = len;
      rec[2] = h == 0 ? none : (h - 1) / 2;
      if (l < L - 1) {
        const uint32_t z = Z[h];
        rec[3] = z ? 2 * h + 1 : none;
        rec[4] = (len - z) ? 2 * h + 2 : none;
      } else {
        rec[3] = rec[4] = none;
      }
    }
  }
  if (ib == 4) {
    uint32_t* o = (uint32_t*)out + 5 * h;
    for (int k = 0; k < 5; ++k) o[k] = (uint32_t)rec[k];
  } else {
    uint64_t* o = (uint64_t*)out + 5 * h;
    for (int k = 0; k < 5; ++k) o[k] = rec[k];
  }
}

// The sequence as the passes read it, on a 32-byte boundary in at most 4 bytes
// a symbol: 8-byte symbols keep their low half (levels <= 24), a sequence that
// does not start on a 32-byte boundary is moved, so that the row loads apply,
// and symbols of fewer bits than there are levels are widened: a digit is
// taken from several packed symbols at once and has to lie inside its own.
template <typename T, typename U>
__global__ void repack_kernel(const T* __restrict__ s, uint64_t n, U* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = (U)s[i];
}

// ------------------------------------------------------------------ host

static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

template <typename T>
static void launch_max(const void* s, uint64_t n, unsigned long long* out, cudaStream_t st) {
  unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 8);
  if (grid == 0) grid = 1;
  max_kernel<T><<<grid, 256, 0, st>>>((const T*)s, n, out);
}

template <typename T, typename U>
static void launch_repack(const void* s, uint64_t n, void* out, cudaStream_t st) {
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 16);
  repack_kernel<T, U><<<grid, 256, 0, st>>>((const T*)s, n, (U*)out);
}

#define WTG_DISPATCH(eb, fn, ...)                       \
  switch (eb) {                                         \
    case 1: fn<uint8_t>(__VA_ARGS__); break;            \
    case 2: fn<uint16_t>(__VA_ARGS__); break;           \
    case 4: fn<uint32_t>(__VA_ARGS__); break;           \
    default: fn<uint64_t>(__VA_ARGS__); break;          \
  }

// host memory the device copies to and from without staging (page-locked or
// registered)
bool host_page_locked(const void* p) {
  cudaPointerAttributes pa{};
  if (cudaPointerGetAttributes(&pa, p) != cudaSuccess) {
    cudaGetLastError();  // clear the query's error
    return false;
  }
  return pa.type == cudaMemoryTypeHost;
}

int tree_levels_from_max(TreeImpl& t, const void* d_seq, uint64_t n, int eb, int* levels) {
  cudaStream_t s = t.stream;
  int rc;
  if ((rc = t.scratch.ensure(sizeof(unsigned long long), s))) return rc;
  WTG_CK(cudaMemsetAsync(t.scratch.p, 0, sizeof(unsigned long long), s));
  if (n) {
    WTG_DISPATCH(eb, launch_max, d_seq, n, t.scratch.as<unsigned long long>(), s);
    count_launch();
    WTG_CK(cudaGetLastError());
  }
  unsigned long long mx = 0;
  WTG_CK(cudaMemcpyAsync(&mx, t.scratch.p, sizeof(mx), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));
  if (mx < 1) mx = 1;
  *levels = (int)hi64(mx) + 1;  // wt_int_par.hpp:385-395 (x starts at 1)
  return WTG_OK;
}

int tree_build(TreeImpl& t, const void* d_seq, uint64_t n, int eb, int L, uint32_t flags) {
  cudaStream_t s = t.stream;
  int rc;
  t.n = n;
  t.levels = L;
  t.elem_bytes = eb;
  t.flags = flags;
  t.bit_words = (n * (uint64_t)L + 63) / 64;
  t.node_tables.ok = t.level_args.ok = t.fm_steps.ok = false;
  ++t.gen;
  const uint64_t heap = 1ull << L;  // heap ids 0 .. 2^L - 2, plus one pad entry

  const uint32_t nchunks = (uint32_t)((n + CHUNK - 1) / CHUNK);
  const int cpw = count_cpw(nchunks);
  const uint32_t tc = LV_WARPS * cpw, tiles = (nchunks + tc - 1) / tc;
  const int groups = n ? (L + 3) / 4 : 0;  // all but the last of four levels
  // the error word, and the look-back state per group: 16 arrays of tile words, a counter
  const uint64_t group_words = 16ull * tiles + 1;
  const size_t err_bytes = 16 + groups * group_words * sizeof(uint64_t);
  if ((rc = t.err.ensure(err_bytes, s))) return rc;
  WTG_CK(cudaMemsetAsync(t.err.p, 0, err_bytes, s));
  t.err.elsewhere = false;
  uint32_t* d_err = t.err.arm(s, s);
  uint64_t* const group_status = t.err.as<uint64_t>() + 2;

  // every string's edge words are ORed in
  if ((rc = t.bits.ensure((t.bit_words + 2) * sizeof(uint64_t), s))) return rc;
  WTG_CK(cudaMemsetAsync(t.bits.p, 0, (t.bit_words + 2) * sizeof(uint64_t), s));
  // per-node tables [Z | C]
  if ((rc = t.zeros.ensure(2 * heap * sizeof(uint32_t), s))) return rc;
  uint32_t* Z = t.zeros.as<uint32_t>();
  uint32_t* C = Z + heap;
  if (n == 0) WTG_CK(cudaMemsetAsync(Z, 0, 2 * heap * sizeof(uint32_t), s));
  else if (L == 1) WTG_CK(cudaMemsetAsync(C, 0, sizeof(uint32_t), s));  // the root (otherwise the first node pass)

  // When the rank table goes to page-locked host memory during the build,
  // the rank/select pass follows the levels, and the rank entries whose bits
  // are final are copied while the later levels are built (a copy to pageable
  // memory would hold the host until it ends); otherwise it is one launch
  // after the last pass.
  const bool rs_by_level = t.host_rank && (flags & WTG_RANK) && n && host_page_locked(t.host_rank);
  if (flags) {
    if ((rc = bv_prepare(t.bv, t.bits.as<uint64_t>(), n * (uint64_t)L, flags, s))) return rc;
  }
  uint64_t rank_copied = 0;  // superblocks whose rank entries were sent
  auto copy_rank = [&]() -> int {
    const uint64_t to = bv_superblocks_done(t.bv);
    if (to <= rank_copied) return WTG_OK;
    WTG_CK(cudaEventRecord(t.copy_ev, s));
    WTG_CK(cudaStreamWaitEvent(t.copy_stream, t.copy_ev, 0));
    WTG_CK(cudaMemcpyAsync(t.host_rank + 2 * rank_copied, t.bv.rank.as<uint64_t>() + 2 * rank_copied,
                           (to - rank_copied) * 16, cudaMemcpyDeviceToHost, t.copy_stream));
    rank_copied = to;
    return WTG_OK;
  };
  if (n) {
    // sequence buffers: what the groups after the first read
    auto bytes_of = [&](int bits_left) { return bits_left > 16 ? 4 : bits_left > 8 ? 2 : 1; };
    const int width = L > 8 * eb ? bytes_of(L) : std::min(eb, 4);
    const bool repack = eb != width || (uintptr_t)d_seq % 32;
    size_t lvl_bytes[2] = {0, repack ? n * width : 0};
    for (int g = 0, sb = width; g + 1 < groups; ++g) {
      sb = std::min(sb, bytes_of(L - 4 * g - 4));
      lvl_bytes[g & 1] = std::max<size_t>(lvl_bytes[g & 1], n * sb);
    }
    DevLayout lay;
    const size_t at_pre = lay.add(((uint64_t)nchunks + 1) * 16 * sizeof(uint32_t));
    const size_t at_cnode = lay.add(((uint64_t)nchunks + 1) * sizeof(uint32_t));
    const size_t at_rec = lay.add((1ull << (4 * (groups - 1))) * REC * sizeof(uint32_t));
    const size_t at_lvl[2] = {lay.add(lvl_bytes[0]), lay.add(lvl_bytes[1])};
    if ((rc = t.work.ensure(lay.bytes, s))) return rc;
    uint8_t* const work = t.work.as<uint8_t>();
    uint32_t* const chunkpre = (uint32_t*)(work + at_pre);
    uint32_t* const cnode = (uint32_t*)(work + at_cnode);
    uint32_t* const rec = (uint32_t*)(work + at_rec);
    void* const lvl[2] = {work + at_lvl[0], work + at_lvl[1]};
    const void* src = d_seq;
    int sb = eb;
    bool waited = t.in_pieces == 0;
    auto wait_pieces = [&]() -> int {
      for (int i = 0; i < t.in_pieces && !waited; ++i) WTG_CK(cudaStreamWaitEvent(s, t.in_ev[i], 0));
      waited = true;
      return WTG_OK;
    };
    if (repack) {
      sb = width;
      if ((rc = wait_pieces())) return rc;
      if (eb != width) {
        if (eb == 8) launch_repack<uint64_t, uint32_t>(d_seq, n, lvl[1], s);
        else if (eb == 2) launch_repack<uint16_t, uint32_t>(d_seq, n, lvl[1], s);
        else if (width == 2) launch_repack<uint8_t, uint16_t>(d_seq, n, lvl[1], s);
        else launch_repack<uint8_t, uint32_t>(d_seq, n, lvl[1], s);
        count_launch();
        WTG_CK(cudaGetLastError());
      } else {
        WTG_CK(cudaMemcpyAsync(lvl[1], d_seq, n * sb, cudaMemcpyDeviceToDevice, s));
      }
      src = lvl[1];
    }
    for (int g = 0; g < groups; ++g) {
      const int l = 4 * g;
      const bool scatter = g + 1 < groups;
      LevelGroup a{};
      a.tau = scatter ? 4 : L - l;
      a.scatter = scatter;
      a.src_bytes = sb;
      a.dst_bytes = scatter ? std::min(sb, bytes_of(L - l - 4)) : 0;
      a.pass.src = src;
      a.pass.n = n;
      a.pass.ds = L - l - a.tau;
      a.pass.level = l;
      a.pass.nchunks = nchunks;
      a.pass.nodes = 1u << l;
      a.pass.Cl = C + ((1ull << l) - 1);
      a.pass.chunkpre = chunkpre;
      a.pass.cnode = cnode;
      a.pass.rec = rec;
      a.pass.bits = t.bits.as<uint32_t>();
      a.pass.err = d_err;
      if (scatter) a.pass.dst = lvl[g & 1];
      a.C = C;
      a.Z = Z;
      a.chunkpre = chunkpre;
      a.cnode = cnode;
      a.rec = rec;
      a.cpw = cpw;
      a.counter = reinterpret_cast<uint32_t*>(group_status + g * group_words);
      a.status = group_status + g * group_words + 1;
      a.sstride = tiles;
      const int tb = scatter ? 4 : a.tau - 1;  // digit bits counted
      if (tb > 0) {
        prof_begin(PROF_HIST, s);
        if (!waited) {
          // each piece of the input is counted once its copy has landed; the
          // passes after it see the whole input
          uint32_t done = 0;
          for (int i = 0; i < t.in_pieces; ++i) {
            WTG_CK(cudaStreamWaitEvent(s, t.in_ev[i], 0));
            const uint64_t have = std::min<uint64_t>(n, ((uint64_t)i + 1) * t.in_piece_symbols);
            const uint32_t to = have == n ? tiles : (uint32_t)(have / ((uint64_t)tc * CHUNK));
            if (to <= done) continue;
            if (done) WTG_CK(cudaMemsetAsync(a.counter, 0, sizeof(uint32_t), s));
            if ((rc = launch_count(a, done, to, s))) return rc;
            done = to;
          }
          waited = true;
        } else if ((rc = launch_count(a, 0, tiles, s))) {
          return rc;
        }
        prof_end(PROF_HIST, s);
        prof_begin(PROF_TABLES, s);
        if ((rc = launch_nodes(a, s))) return rc;
        prof_end(PROF_TABLES, s);
      }
      if ((rc = wait_pieces())) return rc;
      prof_begin(scatter ? PROF_LEVEL : PROF_LEVEL_LAST, s);
      if ((rc = launch_pass(a, s))) return rc;
      prof_end(scatter ? PROF_LEVEL : PROF_LEVEL_LAST, s);
      src = a.pass.dst;
      sb = a.dst_bytes;
      const int done_levels = l + a.tau;
      if (t.host_bits) {
        // words holding only bits of these levels are final now; the word
        // shared with the next level goes with it
        const uint64_t w_lo = ((uint64_t)l * n) >> 6;
        const uint64_t w_hi = done_levels == L ? t.bit_words : ((uint64_t)done_levels * n) >> 6;
        if (w_hi > w_lo) {
          WTG_CK(cudaEventRecord(t.copy_ev, s));
          WTG_CK(cudaStreamWaitEvent(t.copy_stream, t.copy_ev, 0));
          WTG_CK(cudaMemcpyAsync(t.host_bits + w_lo, t.bits.as<uint64_t>() + w_lo, (w_hi - w_lo) * 8,
                                 cudaMemcpyDeviceToHost, t.copy_stream));
        }
      }
      if (rs_by_level && done_levels < L) {
        if ((rc = bv_pass_to(t.bv, (uint64_t)done_levels * n, d_err, s))) return rc;
        if ((rc = copy_rank())) return rc;
      }
    }
  }

  // rank / select over the concatenated bitvector
  if (flags) {
    if ((rc = bv_pass_to(t.bv, n * (uint64_t)L, d_err, s))) return rc;
    // the select finishing kernels run beside the copy of the (last) rank entries
    if (t.host_rank && (flags & WTG_RANK) && (rc = copy_rank())) return rc;
    if ((rc = bv_finish(t.bv, d_err, s))) return rc;
  }
  return WTG_OK;
}

int tree_nodes(TreeImpl& t, int ib, uint64_t n_entries, void* d_out) {
  cudaStream_t s = t.stream;
  if (n_entries == 0) return WTG_OK;
  const uint64_t heap = 1ull << t.levels;
  uint32_t* Z = t.zeros.as<uint32_t>();
  unsigned grid = (unsigned)((n_entries + 255) / 256);
  node_kernel<<<grid, 256, 0, s>>>(Z + heap, Z, t.levels, t.n, n_entries, ib, d_out);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

void tree_release(TreeImpl& t) {
  cudaStream_t s = t.stream;
  if (t.copy_stream) {
    cudaStreamSynchronize(t.copy_stream);
    cudaStreamDestroy(t.copy_stream);
    t.copy_stream = nullptr;
  }
  if (t.copy_ev) cudaEventDestroy(t.copy_ev);
  t.copy_ev = nullptr;
  if (t.in_stream) {
    cudaStreamSynchronize(t.in_stream);
    cudaStreamDestroy(t.in_stream);
    t.in_stream = nullptr;
  }
  for (cudaEvent_t& e : t.in_ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  t.in_pieces = 0;
  lsel_detach_all(t);
  t.seq.release(s);
  t.bits.release(s);
  t.zeros.release(s);
  t.work.release(s);
  t.scan_tmp.release(s);
  t.err.release(s);
  t.level_args.release(s);
  t.node_tables.release(s);
  t.fm_steps.release(s);
  t.scratch.release(s);
  t.nodes.release(s);
  t.qbuf.release(s);
  t.qout.release(s);
  bv_release(t.bv, s);
}

}  // namespace wtg
