// wtg_sa.cu -- suffix array and BWT of a byte text on the GPU: the first two
// steps of the reference's FM-index construction (fm-index/par/WT.C:33-41:
// divsufsort, then bwt[i] = s[SA[i] - 1], or s[n - 1] where SA[i] = 0).
//
// Prefix doubling (Manber & Myers, "Suffix arrays: a new method for on-line
// string searches", 1993) over LSD radix sorts (wtg_radix.cuh):
//   * the text's distinct bytes get codes 1..sigma (0 = past the end); a
//     suffix's first K characters, read as a number in base sigma + 1, are
//     its initial key, so key order is the order of the K-character prefixes
//     (a prefix cut by the end sorts first).  K follows from the order-0
//     entropy: enough characters to tell most suffixes apart, in whole 8-bit
//     sort passes;
//   * after a sort, rank[i] = the suffix-array position of the first slot of
//     suffix i's group (suffixes with equal keys); while groups of several
//     suffixes remain, only their members are re-keyed by
//     (rank[i], rank[i + h] + 1 or 0 past the end) and re-sorted, and h
//     doubles (finished groups are never touched again).
// The sort is stable and every rank is a function of the key, so the result
// is the unique suffix order, the same array divsufsort gives.
#include <algorithm>
#include <cmath>
#include <vector>

#include "wtg_internal.cuh"
#include "wtg_hist.cuh"
#include "wtg_radix.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(sa)

namespace {

constexpr int SA_THREADS = 256;
constexpr int SA_WARPS = SA_THREADS / 32;

// counts of adjacent code pairs over a sample of the text (small alphabets)
constexpr int PAIR_SIGMA = 32;
constexpr uint64_t PAIR_SAMPLE = 1ull << 18;
__global__ void pair_hist_kernel(const uint8_t* __restrict__ s, uint64_t n, const uint16_t* __restrict__ code,
                                 uint64_t step, uint32_t* __restrict__ hist) {
  const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * step;
  if (i + 1 < n) atomicAdd(&hist[(code[s[i]] - 1) * PAIR_SIGMA + code[s[i + 1]] - 1], 1u);
}

// key[i] = s[i .. i + K) as K digits in base B = sigma + 1, codes 1..sigma, 0
// past the end.  A block puts the codes of its positions in shared memory,
// then every four consecutive ones as one number, so a key is K / 4
// multiply-adds (a load and a shift per character took 1.9 ms for 2^27).
constexpr int KEY_TILE = 2048;  // positions per block
__global__ void __launch_bounds__(SA_THREADS)
    init_keys_kernel(const uint8_t* __restrict__ s, uint64_t n, const uint16_t* __restrict__ code_g, uint64_t B, int K,
                     uint64_t* __restrict__ key) {
  __shared__ uint16_t code[256];
  __shared__ uint16_t c[KEY_TILE + 64 + 4];
  __shared__ uint64_t quad[KEY_TILE + 64];
  for (uint32_t i = threadIdx.x; i < 256; i += SA_THREADS) code[i] = code_g[i];
  __syncthreads();
  const uint64_t i0 = (uint64_t)blockIdx.x * KEY_TILE;
  for (uint32_t j = threadIdx.x; j < KEY_TILE + 64 + 4; j += SA_THREADS)
    c[j] = i0 + j < n ? code[s[i0 + j]] : (uint16_t)0;
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < KEY_TILE + 64; j += SA_THREADS)
    quad[j] = (((uint64_t)c[j] * B + c[j + 1]) * B + c[j + 2]) * B + c[j + 3];
  __syncthreads();
  const uint64_t B4 = B * B * B * B;
  for (uint32_t j = threadIdx.x; j < KEY_TILE && i0 + j < n; j += SA_THREADS) {
    uint64_t k = 0;
    int t = 0;
    for (; t + 4 <= K; t += 4) k = k * B4 + quad[j + t];
    for (; t < K; ++t) k = k * B + c[j + t];
    key[i0 + j] = k;
  }
}

// Doubling rounds work on the active list: the suffix-array positions
// act[0..m) (ascending) of the suffixes whose group still holds more than
// one suffix.  A group occupies consecutive positions, its members share
// rank = the position of the group's first slot, and sorting the active
// suffixes by (rank, rank of the suffix h on) lays the groups out in
// position order again, so the k-th sorted suffix goes to position act[k].

// key of active suffix k: (its rank, rank[i + h] + 1, or 0 past the end) for
// i = sa[act[k]]
__global__ void active_keys_kernel(const uint32_t* __restrict__ act, const uint32_t* __restrict__ act_rank,
                                   const uint32_t* __restrict__ sa, const uint32_t* __restrict__ rank, uint64_t m,
                                   uint64_t n, uint64_t h, int B, uint64_t* __restrict__ key,
                                   uint32_t* __restrict__ val) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = sa[act[k]];
    const uint64_t sec = i + h < n ? (uint64_t)rank[i + h] + 1 : 0;
    key[k] = ((uint64_t)act_rank[k] << B) | sec;
    val[k] = i;
  }
}

// After a sort of the m active pairs, in one launch (a look-back over two
// fields: the number of still-shared suffixes before a tile, and the last
// run start before it): suffix val[k] goes to position act[k]; its rank is
// the position of its run's first key; the suffixes still sharing a run with
// another are compacted into act_next, their ranks beside them.  In round 0
// (FIRST) every suffix is active, act is the identity and val the suffix
// array; with rank_of the rank goes beside the suffix for the binned scatter,
// otherwise to its place.  After a wait that ran out (here, or in the sort
// before) the values are no suffixes in places; those are left out.
// A warp takes 16 rows of 32 keys; run starts are one ballot a row.
constexpr int ST_ROWS = 16;
constexpr int ST_TILE = SA_WARPS * ST_ROWS * 32;

template <bool FIRST>
__global__ void __launch_bounds__(SA_THREADS)
    settle_kernel(const uint64_t* __restrict__ key, const uint32_t* __restrict__ val, const uint32_t* __restrict__ act,
                  uint64_t m, uint64_t n, uint32_t* __restrict__ sa, uint32_t* __restrict__ rank, uint32_t* __restrict__ rank_of,
                  uint32_t* __restrict__ act_next, uint32_t* __restrict__ act_rank_next,
                  uint32_t* __restrict__ shared_total, uint64_t* status_cnt, uint64_t* status_head, uint32_t* counter,
                  uint32_t* err) {
  __shared__ uint32_t s_tile, s_cnt_before, s_head_before;
  __shared__ uint32_t ws[SA_WARPS], wh[SA_WARPS];
  if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t le = 0xffffffffu >> (31 - lane), lt = le >> 1;
  const uint64_t t0 = (uint64_t)tile * ST_TILE;
  const uint64_t k0 = t0 + warp * (ST_ROWS * 32) + lane;
  // S[j]: run starts of row j; keys from m on count as starts
  uint32_t S[ST_ROWS + 1];
  {
    uint64_t x[ST_ROWS + 1];
#pragma unroll
    for (int j = 0; j <= ST_ROWS; ++j) {
      const uint64_t k = k0 + 32 * j;
      x[j] = (j < ST_ROWS || lane == 0) && k < m ? key[k] : 0;
    }
    uint64_t last = k0 - lane > 0 && k0 - lane <= m ? key[k0 - lane - 1] : 0;  // the key before the row
#pragma unroll
    for (int j = 0; j <= ST_ROWS; ++j) {
      const uint64_t k = k0 + 32 * j;
      uint64_t prev = __shfl_up_sync(0xffffffffu, x[j], 1);
      if (lane == 0) prev = last;
      S[j] = __ballot_sync(0xffffffffu, k >= m || k == 0 || prev != x[j]);
      last = __shfl_sync(0xffffffffu, x[j], 31);
    }
  }
  // U[j]: suffixes alone in their run; head: 1 + index of the last run start
  uint32_t cnt = 0, head = 0;
#pragma unroll
  for (int j = 0; j < ST_ROWS; ++j) {
    const uint64_t r0 = k0 - lane + 32 * j;
    const uint32_t in = r0 >= m ? 0u : m - r0 >= 32 ? 0xffffffffu : (1u << (m - r0)) - 1u;
    const uint32_t alone = S[j] & __funnelshift_r(S[j], S[j + 1], 1);
    cnt += __popc(in & ~alone);
    const uint32_t st = S[j] & in;
    if (st) head = (uint32_t)r0 + 32 - __clz(st);
  }
  if (lane == 0) {
    ws[warp] = cnt;
    wh[warp] = head;
  }
  __syncthreads();
  uint32_t total = 0, last = 0;
  for (int w = 0; w < SA_WARPS; ++w) {
    total += ws[w];
    last = max(last, wh[w]);
  }
  if (warp == 0) {
    uint64_t before = 0;
    if (tile > 0) {
      if (lane == 0) lb_publish(status_cnt, tile, LB_FLAG_AGG, total);
      before = lb_lookback_warp(status_cnt, tile, err);
    }
    if (lane == 0) {
      lb_publish(status_cnt, tile, LB_FLAG_INC, before + total);
      s_cnt_before = (uint32_t)before;
      if (t0 + ST_TILE >= m) *shared_total = (uint32_t)before + total;
    }
  } else if (warp == 1) {
    // the last run start before the tile: the nearest predecessor that has
    // one names it (position 0 is a start, so one always does)
    uint32_t h = 0;
    if (lane == 0) lb_publish(status_head, tile, last ? LB_FLAG_INC : LB_FLAG_AGG, last);
    if (tile > 0) {
      for (int64_t at = (int64_t)tile - 1; at >= 0; at -= 32) {
        const int64_t p = at - lane;
        uint64_t v = LB_FLAG_AGG;
        if (p >= 0) {
          uint32_t spins = 0, ns = 32;
          while (((v = lb_load(status_head, (uint64_t)p)) >> 62) == 0) {
            if (++spins > c_wait_limit[0]) {
              atomicCAS(err, 0u, (uint32_t)DERR_LOOKBACK_TIMEOUT);
              v = LB_FLAG_INC | 1;  // (position 0 is a start)
              break;
            }
            __nanosleep(ns);
            if (ns < 1024) ns <<= 1;
          }
        }
        const uint32_t has = __ballot_sync(0xffffffffu, (v >> 62) == 2);
        if (has) {
          h = __shfl_sync(0xffffffffu, (uint32_t)(v & LB_VALUE_MASK), __ffs(has) - 1);
          break;
        }
      }
    }
    if (lane == 0) {
      s_head_before = h;
      // a tile within one run passes the start on: where a run spans many tiles
      // every one of them walked back over all before it (2^26 equal bytes, 2^14
      // tiles: 4.8 ms a launch, 1.4 so)
      if (!last) lb_publish(status_head, tile, LB_FLAG_INC, h);
    }
  }
  __syncthreads();
  uint32_t c = s_cnt_before, h = s_head_before;
  for (uint32_t w = 0; w < warp; ++w) {
    c += ws[w];
    h = max(h, wh[w]);
  }
#pragma unroll
  for (int j = 0; j < ST_ROWS; ++j) {
    const uint64_t r0 = k0 - lane + 32 * j;
    if (r0 >= m) break;
    const uint64_t k = r0 + lane;
    const uint32_t in = m - r0 >= 32 ? 0xffffffffu : (1u << (m - r0)) - 1u;
    const uint32_t shared = in & ~(S[j] & __funnelshift_r(S[j], S[j + 1], 1));
    const uint32_t mine = S[j] & in & le;  // run starts up to this key
    const uint32_t first = (mine ? (uint32_t)r0 + 32 - __clz(mine) : h) - 1;
    if (k < m) {
      const uint32_t pos = FIRST ? (uint32_t)k : act[k];
      const uint32_t r = FIRST ? first : act[first];
      if (FIRST && rank_of) {
        rank_of[k] = r;
      } else {
        const uint32_t i = val[k];
        if (!FIRST) sa[pos] = i;
        if (i < n) rank[i] = r;
      }
      if ((shared >> lane) & 1u) {
        act_next[c + __popc(shared & lt)] = pos;
        act_rank_next[c + __popc(shared & lt)] = r;
      }
    }
    c += __popc(shared);
    const uint32_t st = S[j] & in;
    if (st) h = (uint32_t)r0 + 32 - __clz(st);
  }
}

// rank[i] = r for the pairs of the binned scatter; a block per 2048 pairs, so
// that the blocks in flight stay within a few bins (a grid stride let them
// drift over most of the array: 2.6 ms for 2^27)
constexpr int RSC_PAIRS = 8;
__global__ void __launch_bounds__(256) rank_scatter_kernel(const uint32_t* __restrict__ i, const uint32_t* __restrict__ r,
                                                           uint64_t n, uint32_t* __restrict__ rank) {
  const uint64_t k0 = (uint64_t)blockIdx.x * (256 * RSC_PAIRS) + threadIdx.x;
#pragma unroll
  for (int j = 0; j < RSC_PAIRS; ++j) {
    const uint64_t k = k0 + 256 * j;
    if (k < n) {
      const uint32_t at = i[k];
      if (at < n) rank[at] = r[k];  // (always, but after a failed look-back of the binning)
    }
  }
}

// fm-index/par/WT.C:38-41: bwt[j] = s[SA[j] - 1], or s[n - 1] where SA[j] = 0
__global__ void bwt_kernel(const uint8_t* __restrict__ s, const uint32_t* __restrict__ sa, uint64_t n,
                           uint8_t* __restrict__ bwt) {
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t p = sa[j];
    bwt[j] = s[p ? p - 1 : n - 1];
  }
}

// The same from the text's codes in half a byte each (alphabets of at most 16
// bytes): the gather is bound by the sectors that L2 does not hold, and the
// codes of 2^27 symbols are 67 MB of its 126 (the text alone fills it).  2^27
// DNA codes: 0.55 ms with the packing, 1.27 from the text.  Below 2^25 symbols
// L2 holds the text.
constexpr uint64_t PACK_MIN = 1ull << 25;
__global__ void __launch_bounds__(256) pack_codes_kernel(const uint8_t* __restrict__ s, uint64_t n,
                                                         const uint16_t* __restrict__ code,
                                                         uint32_t* __restrict__ packed) {
  __shared__ uint8_t c[256];
  c[threadIdx.x] = (uint8_t)(code[threadIdx.x] - 1);
  __syncthreads();
  const bool words = ((uintptr_t)s & 7) == 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < (n + 7) / 8; k += stride) {
    uint64_t w = 0;
    if (words && 8 * k + 8 <= n) {
      w = __ldg(reinterpret_cast<const uint64_t*>(s) + k);
    } else {
      for (uint32_t e = 0; e < 8 && 8 * k + e < n; ++e) w |= (uint64_t)s[8 * k + e] << (8 * e);
    }
    uint32_t x = 0;
#pragma unroll
    for (uint32_t e = 0; e < 8; ++e) x |= (uint32_t)(c[(w >> (8 * e)) & 0xFFu] & 15u) << (4 * e);
    packed[k] = x;
  }
}
constexpr int BWT_PER = 8;
__global__ void __launch_bounds__(256) bwt_packed_kernel(const uint8_t* __restrict__ packed,
                                                         const uint16_t* __restrict__ code,
                                                         const uint32_t* __restrict__ sa, uint64_t n,
                                                         uint8_t* __restrict__ bwt) {
  __shared__ uint8_t byte_of[16];
  const uint32_t mine = code[threadIdx.x];
  if (mine) byte_of[mine - 1] = (uint8_t)threadIdx.x;
  __syncthreads();
  const uint64_t j0 = (uint64_t)blockIdx.x * (256 * BWT_PER) + threadIdx.x;
  uint32_t p[BWT_PER];
#pragma unroll
  for (int k = 0; k < BWT_PER; ++k) {
    const uint64_t j = j0 + 256 * k;
    const uint32_t v = j < n ? __ldg(sa + j) : 1u;
    p[k] = v ? v - 1 : (uint32_t)(n - 1);
  }
#pragma unroll
  for (int k = 0; k < BWT_PER; ++k) p[k] = (__ldg(packed + (p[k] >> 1)) >> (4 * (p[k] & 1))) & 15u;
#pragma unroll
  for (int k = 0; k < BWT_PER; ++k)
    if (j0 + 256 * k < n) bwt[j0 + 256 * k] = byte_of[p[k]];
}

int bit_width64(uint64_t x) { return x ? 64 - __builtin_clzll(x) : 0; }

unsigned grid_for(uint64_t n) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, 152ull * 16));
}

}  // namespace

// Scratch of one suffix-array run, released when it ends.
struct SaScratch {
  DevBuf key[2], val[2], rank, sa_own, act[2], act_rank, hist, status, err, small;
  uint32_t* sa = nullptr;  // the suffix array: in the caller's array, or sa_own
  cudaStream_t s;
  explicit SaScratch(cudaStream_t st) : s(st) {}
  ~SaScratch() {
    for (auto* b : {&key[0], &key[1], &val[0], &val[1], &rank, &sa_own, &act[0], &act[1], &act_rank, &hist,
                    &status, &err, &small})
      b->release(s);
  }
};

// val: the two value buffers (round 0 sorts into the suffix array itself)
static int sort_pairs(SaScratch& x, uint64_t n, int bits, bool iota, uint32_t* const val[2], int& cur) {
  uint64_t* const key[2] = {x.key[0].as<uint64_t>(), x.key[1].as<uint64_t>()};
  const int passes = (bits + 7) / 8;
  int rc;
  if ((rc = x.status.ensure(radix_status_bytes(n, passes), x.s))) return rc;
  return radix_sort_pairs<uint64_t>(key, val, n, 0, passes, iota, x.hist.as<uint32_t>(), x.status.as<uint8_t>(),
                                    x.err.as<uint32_t>(), cur, x.s);
}

// From so many suffixes on, round 0's ranks reach their places in two steps:
// (suffix, rank) pairs binned by the suffix's top byte, then scattered within
// a bin's part of the rank array, which stays in L2.  Scattering straight to
// 2^27 places costs a DRAM sector read and write for 4 bytes (5.5 ms, binned
// 0.9 ms); below 2^24 the rank array fits in half of the L2 anyway.
constexpr uint64_t RANK_BIN_MIN = 1ull << 24;

// after a sort of the m active pairs (in key[cur] / val[cur]): place them,
// refresh their ranks and compact the still-shared ones into act[ac ^ 1];
// first: round 0, all suffixes
static int settle_round(SaScratch& x, uint64_t m, uint64_t n, bool first, const uint32_t* val, int cur, int& ac,
                        uint64_t* m_next) {
  int rc;
  const uint64_t tiles = (m + ST_TILE - 1) / ST_TILE;
  if ((rc = x.status.ensure((2 * tiles + 1) * sizeof(uint64_t), x.s))) return rc;
  WTG_CK(cudaMemsetAsync(x.status.p, 0, (2 * tiles + 1) * sizeof(uint64_t), x.s));
  uint64_t* st = x.status.as<uint64_t>();
  uint32_t* total = x.small.as<uint32_t>();
  const bool binned = first && m >= RANK_BIN_MIN;
  // the key buffers are free once the keys are read: the other one takes the ranks
  uint32_t* rank_of = binned ? x.key[cur ^ 1].as<uint32_t>() : nullptr;
  auto* const f = first ? settle_kernel<true> : settle_kernel<false>;
  f<<<(unsigned)tiles, SA_THREADS, 0, x.s>>>(
      x.key[cur].as<uint64_t>(), val, first ? nullptr : x.act[ac].as<uint32_t>(), m, n, x.sa, x.rank.as<uint32_t>(),
      rank_of, x.act[ac ^ 1].as<uint32_t>(), x.act_rank.as<uint32_t>(), total, st + 1, st + 1 + tiles,
      reinterpret_cast<uint32_t*>(st), x.err.as<uint32_t>());
  count_launch();
  WTG_CK(cudaGetLastError());
  uint32_t h[2] = {0, 0};
  WTG_CK(cudaMemcpyAsync(&h[0], total, sizeof(uint32_t), cudaMemcpyDeviceToHost, x.s));
  WTG_CK(cudaMemcpyAsync(&h[1], x.err.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, x.s));
  WTG_CK(cudaStreamSynchronize(x.s));
  if (h[1]) return fail(WTG_ERR_TIMEOUT, "suffix array: a scan wait timed out");
  if (binned && h[0]) {  // (without shared suffixes no rank is read)
    // bin by the top byte of the suffix numbers
    const int byte = (bit_width64(m - 1) - 1) / 8;
    uint32_t* const k2[2] = {x.sa, x.val[0].as<uint32_t>()};  // (the first is only read)
    uint32_t* const v2[2] = {rank_of, x.key[cur].as<uint32_t>()};
    int c2 = 0;
    if ((rc = x.status.ensure(radix_status_bytes(m, 1), x.s))) return rc;
    if ((rc = radix_sort_pairs<uint32_t>(k2, v2, m, 8 * byte, 1, false, x.hist.as<uint32_t>(), x.status.as<uint8_t>(),
                                         x.err.as<uint32_t>(), c2, x.s)))
      return rc;
    rank_scatter_kernel<<<(unsigned)((m + 256 * RSC_PAIRS - 1) / (256 * RSC_PAIRS)), 256, 0, x.s>>>(k2[c2], v2[c2], m, x.rank.as<uint32_t>());
    count_launch();
    WTG_CK(cudaGetLastError());
  }
  ac ^= 1;
  *m_next = h[0];
  return WTG_OK;
}

// Whether the suffix array can be made in the caller's array: device memory on
// 4 bytes, apart from the BWT (which is written while it is read).  Others get a
// copy at the end.
static bool usable_in_place(const uint32_t* d_sa, const uint8_t* d_bwt, uint64_t n) {
  if ((uintptr_t)d_sa % 4) return false;
  const uintptr_t a = (uintptr_t)d_sa, b = (uintptr_t)d_bwt;
  if (d_bwt && a < b + n && b < a + 4 * n) return false;
  cudaPointerAttributes pa{};
  if (cudaPointerGetAttributes(&pa, d_sa) != cudaSuccess) {
    cudaGetLastError();  // clear the query's error
    return false;
  }
  return pa.type == cudaMemoryTypeDevice;
}

int suffix_array_device(const uint8_t* d_text, uint64_t n, uint32_t* d_sa, uint8_t* d_bwt, int* rounds,
                        cudaStream_t s) {
  int rc;
  if (rounds) *rounds = 0;
  if (n == 0) return WTG_OK;
  if (n >= (1ull << 31)) return fail(WTG_ERR_INVALID, "suffix array: n must be below 2^31 (32-bit entries)");
  SaScratch x(s);
  const bool in_place = d_sa && usable_in_place(d_sa, d_bwt, n);
  if ((rc = x.key[0].ensure(n * 8 + 8, s)) || (rc = x.key[1].ensure(n * 8 + 8, s)) ||
      (rc = x.val[0].ensure(n * 4, s)) || (rc = x.val[1].ensure(n * 4, s)) || (rc = x.rank.ensure(n * 4, s)) ||
      (!in_place && (rc = x.sa_own.ensure(n * 4, s))) || (rc = x.act[0].ensure(n * 4, s)) || (rc = x.act[1].ensure(n * 4, s)) ||
      (rc = x.act_rank.ensure(n * 4, s)) ||
      (rc = x.hist.ensure(RS_MAX_PASSES * RS_RADIX * 4, s)) || (rc = x.err.ensure(4, s)) ||
      (rc = x.small.ensure(2048 + PAIR_SIGMA * PAIR_SIGMA * 4, s)))
    return rc;
  WTG_CK(cudaMemsetAsync(x.err.p, 0, 4, s));
  // alphabet: codes 1..sigma in byte order
  uint32_t* d_hist = x.small.as<uint32_t>();
  WTG_CK(cudaMemsetAsync(d_hist, 0, 256 * 4, s));
  byte_hist_kernel<uint32_t><<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + 8191) / 8192, 152 * 4)), 512, 0, s>>>(
      d_text, n, d_hist);
  count_launch();
  WTG_CK(cudaGetLastError());
  uint32_t hist[256];
  WTG_CK(cudaMemcpyAsync(hist, d_hist, sizeof(hist), cudaMemcpyDeviceToHost, s));
  WTG_CK(cudaStreamSynchronize(s));
  uint16_t code[256];  // 1..sigma, sigma <= 256
  int sigma = 0;
  double H = 0;  // bits per character, order 0
  for (int c = 0; c < 256; ++c) {
    code[c] = hist[c] ? (uint16_t)++sigma : 0;
    if (hist[c]) H -= (double)hist[c] / n * std::log2((double)hist[c] / n);
  }
  uint16_t* d_code = (uint16_t*)(x.small.as<uint32_t>() + 256);
  WTG_CK(cudaMemcpyAsync(d_code, code, sizeof(code), cudaMemcpyHostToDevice, s));
  if (sigma > 1 && sigma <= PAIR_SIGMA && n >= 4 * PAIR_SAMPLE) {
    // of a small alphabet the characters are told apart by their context as
    // well: H becomes the entropy of a character after another, from a sample
    uint32_t* d_pair = x.small.as<uint32_t>() + 512;
    std::vector<uint32_t> pair(PAIR_SIGMA * PAIR_SIGMA);
    WTG_CK(cudaMemsetAsync(d_pair, 0, pair.size() * 4, s));
    pair_hist_kernel<<<(unsigned)(PAIR_SAMPLE / 256), 256, 0, s>>>(d_text, n, d_code, n / PAIR_SAMPLE, d_pair);
    count_launch();
    WTG_CK(cudaGetLastError());
    WTG_CK(cudaMemcpyAsync(pair.data(), d_pair, pair.size() * 4, cudaMemcpyDeviceToHost, s));
    WTG_CK(cudaStreamSynchronize(s));
    double all = 0, H1 = 0;
    for (uint32_t v : pair) all += v;
    for (int a = 0; a < sigma; ++a) {
      double row = 0;
      for (int b = 0; b < sigma; ++b) row += pair[a * PAIR_SIGMA + b];
      for (int b = 0; b < sigma; ++b)
        if (const double v = pair[a * PAIR_SIGMA + b]) H1 -= v / all * std::log2(v / row);
    }
    H = std::min(H, H1);
  }
  // characters of the first key: those that tell suffixes apart with some
  // margin (real texts repeat more than this entropy says), at least 4; then
  // as many as fit in the sort passes these need.  (2^27 DNA codes: 21
  // characters and 7 passes left 19 % of the suffixes to the next round.)
  const double per = std::log2((double)sigma + 1);
  const double want = std::max(4.0, (std::log2((double)n) + 12) / std::max(H, 0.1));
  const int passes = (int)std::min(8.0, std::ceil(want * per / 8));
  int K = 0;
  uint64_t most = 1;  // (sigma + 1)^K <= 2^(8 passes)
  const uint64_t B1 = (uint64_t)sigma + 1;
  const uint64_t lim = passes == 8 ? ~0ull : (1ull << (8 * passes));
  while (K < 60 && most <= lim / B1) {
    most *= B1;
    ++K;
  }
  // round 0: every suffix, keyed by its first K codes
  init_keys_kernel<<<(unsigned)((n + KEY_TILE - 1) / KEY_TILE), SA_THREADS, 0, s>>>(d_text, n, d_code, B1, K,
                                                                                   x.key[0].as<uint64_t>());
  count_launch();
  WTG_CK(cudaGetLastError());
  // the values of the last pass are the suffix array: it is one of the two
  // value buffers, the one that the number of passes ends in
  int cur = 0, ac = 0;
  x.sa = in_place ? d_sa : x.sa_own.as<uint32_t>();
  uint32_t* const val0[2] = {passes & 1 ? x.val[0].as<uint32_t>() : x.sa, passes & 1 ? x.sa : x.val[0].as<uint32_t>()};
  uint32_t* const val[2] = {x.val[0].as<uint32_t>(), x.val[1].as<uint32_t>()};
  if ((rc = sort_pairs(x, n, 8 * passes, true, val0, cur))) return rc;
  uint64_t m = 0;
  if ((rc = settle_round(x, n, n, true, x.sa, cur, ac, &m))) return rc;
  uint64_t h = (uint64_t)K;
  int r = 0;
  const int B = bit_width64(n);               // rank[i + h] + 1 <= n
  const int hi = B + bit_width64(n - 1);      // rank < n
  while (m) {
    active_keys_kernel<<<grid_for(m), 256, 0, s>>>(x.act[ac].as<uint32_t>(), x.act_rank.as<uint32_t>(), x.sa,
                                                   x.rank.as<uint32_t>(), m, n, h, B, x.key[cur].as<uint64_t>(),
                                                   val[cur]);
    count_launch();
    WTG_CK(cudaGetLastError());
    if ((rc = sort_pairs(x, m, hi, false, val, cur))) return rc;
    if ((rc = settle_round(x, m, n, false, val[cur], cur, ac, &m))) return rc;
    h *= 2;
    ++r;
  }
  if (rounds) *rounds = r;
  if (d_sa && !in_place) WTG_CK(cudaMemcpyAsync(d_sa, x.sa, n * 4, cudaMemcpyDeviceToDevice, s));
  if (d_bwt) {
    if (sigma <= 16 && n >= PACK_MIN) {  // (the keys' buffers are free by now)
      pack_codes_kernel<<<grid_for((n + 7) / 8), 256, 0, s>>>(d_text, n, d_code, x.key[0].as<uint32_t>());
      count_launch();
      WTG_CK(cudaGetLastError());
      bwt_packed_kernel<<<(unsigned)((n + 256 * BWT_PER - 1) / (256 * BWT_PER)), 256, 0, s>>>(
          x.key[0].as<uint8_t>(), d_code, x.sa, n, d_bwt);
    } else {
      bwt_kernel<<<grid_for(n), 256, 0, s>>>(d_text, x.sa, n, d_bwt);
    }
    count_launch();
    WTG_CK(cudaGetLastError());
  }
  WTG_CK(cudaStreamSynchronize(s));
  return WTG_OK;
}

}  // namespace wtg
