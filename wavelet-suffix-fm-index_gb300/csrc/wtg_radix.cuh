// wtg_radix.cuh -- stable LSD radix sort of (key, value) pairs on the GPU
// (internal): one launch per 8-bit digit.
//
// The digit histograms of all passes come from one read of the keys.  A pass
// then reads and writes every pair once: a tile of 6144 pairs ranks its
// digits, publishes its digit counts, adds up its predecessors' by a
// decoupled look-back (thread per digit), puts the pairs in digit order in
// shared memory and writes the runs out.  (Adinets & Merrill, "Onesweep: A
// Faster Least Significant Digit Radix Sort for GPUs", 2022.)  The passes
// before this one counted each digit in a launch of its own, scanned 256 x
// tiles counts in another and ranked every pair twice.
//
// A pass over 2^27 pairs of 8 + 4 bytes takes 1.04 ms (3.1 TB/s; 2.05 ms in
// three launches before); it is bound by instruction issue and shared-memory
// latency, 140 warp instructions per 32 pairs.  Measured per pass: 256
// threads of 16 pairs 1.06 ms, 512 of 8 1.11 ms; ranks by match.any 1.43 ms,
// by shared-memory OR 1.30 ms; a test for whole tiles in the loads 1.4 ms (a
// branch around each load); values loaded before the look-back 1.28 ms
// (registers).
#pragma once
#include <type_traits>

#include "wtg_internal.cuh"

namespace wtg {

constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_IPT = 12;                     // pairs per thread
constexpr int RS_TILE = RS_THREADS * RS_IPT;   // 6144
constexpr int RS_CTAS = 2;
constexpr int RS_RADIX = 256;
constexpr int RS_MAX_PASSES = 8;

// hist[pass][digit] of keys' bits [lo + 8 pass, lo + 8 pass + 8)
template <typename K>
__global__ void __launch_bounds__(RS_THREADS)
    radix_hist_kernel(const K* __restrict__ key, uint64_t n, int lo, int passes, uint32_t* __restrict__ hist,
                      const uint32_t* __restrict__ skip) {
  if (skip && *skip) return;
  __shared__ uint32_t h[RS_MAX_PASSES][RS_RADIX];
  for (uint32_t i = threadIdx.x; i < RS_MAX_PASSES * RS_RADIX; i += RS_THREADS) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * RS_THREADS;
  const uint32_t lane = threadIdx.x & 31;
  // whole warps: a digit that all lanes share (the top digits of sorted or
  // skewed keys) is one add; the rest key by key
  const uint64_t whole = n & ~31ull;
  for (uint64_t i = (uint64_t)blockIdx.x * RS_THREADS + threadIdx.x; i < whole; i += stride) {
    const K k = key[i] >> lo;
#pragma unroll
    for (int p = 0; p < RS_MAX_PASSES; ++p) {
      if (p >= passes) break;
      const uint32_t d = (uint32_t)(k >> (8 * p)) & 255u;
      int same;
      __match_all_sync(0xffffffffu, d, &same);
      if (!same) atomicAdd(&h[p][d], 1u);
      else if (lane == 0) atomicAdd(&h[p][d], 32u);
    }
  }
  if (blockIdx.x == 0 && whole + threadIdx.x < n) {
    const K k = key[whole + threadIdx.x] >> lo;
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(uint32_t)(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < (uint32_t)passes * RS_RADIX; j += RS_THREADS) {
    const uint32_t v = (&h[0][0])[j];
    if (v) atomicAdd(&hist[j], v);
  }
}

// exclusive scan of each pass's histogram, in place (block per pass)
static __global__ void __launch_bounds__(RS_RADIX) radix_bases_kernel(uint32_t* __restrict__ hist) {
  __shared__ uint32_t ws[RS_RADIX / 32];
  uint32_t* h = hist + (uint64_t)blockIdx.x * RS_RADIX;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t v = h[threadIdx.x];
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (uint32_t)o) inc += x;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  for (uint32_t k = 0; k < warp; ++k) inc += ws[k];
  h[threadIdx.x] = inc - v;
}

// Status word of a tile and digit: flag in the top two bits, count below.
// 32-bit words hold counts below 2^30.
template <typename S>
struct RadixStatus {
  static constexpr int SHIFT = 8 * sizeof(S) - 2;
  static constexpr S AGG = S(1) << SHIFT, INC = S(2) << SHIFT, MASK = AGG - 1;
};

// the 8-bit digit of a key at bit `shift` (a multiple of 8 for 8-byte keys)
__device__ __forceinline__ uint32_t key_digit(uint64_t k, int shift) {
  return __byte_perm((uint32_t)k, (uint32_t)(k >> 32), 0x4440 + (shift >> 3)) & 255u;
}
__device__ __forceinline__ uint32_t key_digit(uint32_t k, int shift) { return (k >> shift) & 255u; }

// lanes of the warp with the same 8-bit digit (all 32 take part)
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool bit = (d >> b) & 1u;
    const uint32_t v = __ballot_sync(0xffffffffu, bit);
    m &= bit ? v : ~v;
  }
  return m;
}

// One pass.  IOTA: the values are the indices (val is not read).
template <typename K, typename S, bool IOTA>
__global__ void __launch_bounds__(RS_THREADS, RS_CTAS)
    radix_pass_kernel(const K* __restrict__ key, const uint32_t* __restrict__ val, uint64_t n, int shift,
                      const uint32_t* __restrict__ bases, S* status, uint32_t* counter, K* __restrict__ key_out,
                      uint32_t* __restrict__ val_out, uint32_t* err, const uint32_t* __restrict__ skip) {
  if (skip && *skip) return;
  using RS = RadixStatus<S>;
  __shared__ __align__(16) K s_key[RS_TILE];
  __shared__ uint32_t wc[RS_WARPS][RS_RADIX];  // per warp: count, then local base
  __shared__ uint32_t gdelta[RS_RADIX];     // global position - local index (mod 2^32)
  __shared__ uint32_t wsum[RS_WARPS];
  __shared__ uint32_t s_tile;
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(counter, 1u);
  for (uint32_t i = tid; i < RS_WARPS * RS_RADIX; i += RS_THREADS) (&wc[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t tile0 = (uint64_t)tile * RS_TILE;
  const uint32_t tn = (uint32_t)min((uint64_t)RS_TILE, n - tile0);
  const uint32_t off = w * (32 * RS_IPT) + lane;
  const uint32_t lt = (1u << lane) - 1u;
  const K* __restrict__ kp = key + tile0 + off;
  K k[RS_IPT];
  uint32_t rk[RS_IPT];  // rank in the warp among its digit, then local place
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j) k[j] = off + 32 * j < tn ? kp[32 * j] : ~K(0);  // past the end: digit 255
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j) {
    const uint32_t d = key_digit(k[j], shift);
    const uint32_t m = same_digit(d);
    const uint32_t old = wc[w][d];
    rk[j] = old + __popc(m & lt);
    __syncwarp();
    if (!(m & lt)) wc[w][d] = old + __popc(m);
    __syncwarp();
  }
  __syncthreads();
  // thread d: digit d's count in the tile, the warps' local bases, look-back
  uint32_t tot = 0, inc = 0, real = 0;
  volatile S* const st = status + (uint64_t)tile * RS_RADIX + tid;
  if (tid < RS_RADIX) {
#pragma unroll
    for (int x = 0; x < RS_WARPS; ++x) tot += wc[x][tid];
    // the places past the end count as digit 255
    real = tid == 255 ? tot - (RS_TILE - tn) : tot;
    *st = (tile == 0 ? RS::INC : RS::AGG) | (S)real;
    inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= (uint32_t)o) inc += x;
    }
    if (lane == 31) wsum[w] = inc;
  }
  __syncthreads();
  if (tid < RS_RADIX) {
    uint32_t start = inc - tot;
    for (uint32_t x = 0; x < w; ++x) start += wsum[x];
    uint32_t run = start;
#pragma unroll
    for (int x = 0; x < RS_WARPS; ++x) {
      const uint32_t c = wc[x][tid];
      wc[x][tid] = run;
      run += c;
    }
    uint32_t before = 0;
    if (tile > 0) {
      // four predecessors at a time: one by one, each a trip to L2, the walk
      // over the tiles in flight took longer than the tile
      constexpr int AHEAD = 4;
      uint32_t spins = 0, ns = 32;
      int64_t t = (int64_t)tile - 1;
      for (bool done = false; !done;) {
        S v[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q)
          v[q] = t - q >= 0 ? *(volatile const S*)(status + (uint64_t)(t - q) * RS_RADIX + tid) : RS::INC;
        int q = 0;
#pragma unroll
        for (int e = 0; e < AHEAD; ++e) {
          const S flag = v[e] & ~RS::MASK;
          if (done || q < e || !flag) continue;  // past the end, or past one that is not there yet
          before += (uint32_t)(v[e] & RS::MASK);
          done = flag == RS::INC;
          ++q;
        }
        t -= q;
        if (!done && q == 0) {
          if (++spins > c_wait_limit[0]) {
            atomicCAS(err, 0u, (uint32_t)DERR_LOOKBACK_TIMEOUT);
            break;
          }
          if (spins > 8) {
            __nanosleep(ns);
            if (ns < 1024) ns <<= 1;
          }
        }
      }
      *st = RS::INC | (S)(before + real);
    }
    gdelta[tid] = bases[tid] + before - start;
  }
  __syncthreads();
  // into digit order, keys first, then the values through the same room
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j) {
    rk[j] += wc[w][key_digit(k[j], shift)];
    s_key[rk[j]] = k[j];
  }
  __syncthreads();
  uint32_t g[RS_IPT];
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j) {
    const uint32_t i = tid + j * RS_THREADS;
    const K x = s_key[i];
    g[j] = i + gdelta[key_digit(x, shift)];
    if (i >= tn) g[j] = 0xffffffffu;
    if (g[j] < n) key_out[g[j]] = x;  // (always, but for places past the end and a failed look-back)
  }
  __syncthreads();
  uint32_t* const s_val = reinterpret_cast<uint32_t*>(s_key);
  const uint32_t* __restrict__ vp = val + tile0 + off;
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j)
    s_val[rk[j]] = IOTA ? (uint32_t)tile0 + off + 32 * j : (off + 32 * j < tn ? vp[32 * j] : 0u);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < RS_IPT; ++j)
    if (g[j] < n) val_out[g[j]] = s_val[tid + j * RS_THREADS];
}

// Sorts n pairs by key bits [lo, lo + 8 passes), lo a multiple of 8 for 8-byte keys; the pairs are in key[cur] /
// val[cur] and end there (cur flips once per pass).  iota: the values of the
// first pass are the indices.  hist: passes * 256 words, status: its bytes
// from radix_status_bytes; both are scratch.  skip: a device word that, when
// set, leaves the sort out (nothing of its outputs is written).  Asynchronous.
inline uint64_t radix_status_bytes(uint64_t n, int passes) {
  const uint64_t tiles = (n + RS_TILE - 1) / RS_TILE;
  return (uint64_t)passes * (tiles * RS_RADIX * (n < (1ull << 30) ? 4 : 8) + 16);
}

template <typename K, typename S>
int radix_passes(K* const key[2], uint32_t* const val[2], uint64_t n, int lo, int passes, bool iota, uint32_t* hist,
                 uint8_t* status, uint32_t* d_err, int& cur, cudaStream_t s, const uint32_t* skip) {
  const uint32_t tiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
  const uint64_t per = (uint64_t)tiles * RS_RADIX * sizeof(S) + 16;
  for (int p = 0; p < passes; ++p) {
    uint8_t* st = status + p * per;
    uint32_t* counter = reinterpret_cast<uint32_t*>(st);
    S* words = reinterpret_cast<S*>(st + 16);
    uint32_t grid = tiles;
    if (p == 0 && tiles > 1 && test_take_lookback_stall()) {  // tile 0 is never taken, as in bv_prepare
      WTG_CK(cudaMemsetAsync(counter, 1, 1, s));
      --grid;
    }
    if (iota && p == 0)
      radix_pass_kernel<K, S, true><<<grid, RS_THREADS, 0, s>>>(key[cur], val[cur], n, lo, hist, words, counter,
                                                                key[cur ^ 1], val[cur ^ 1], d_err, skip);
    else
      radix_pass_kernel<K, S, false><<<grid, RS_THREADS, 0, s>>>(key[cur], val[cur], n, lo + 8 * p,
                                                                  hist + p * RS_RADIX, words, counter, key[cur ^ 1],
                                                                 val[cur ^ 1], d_err, skip);
    count_launch();
    WTG_CK(cudaGetLastError());
    cur ^= 1;
  }
  return WTG_OK;
}

template <typename K>
int radix_sort_pairs(K* const key[2], uint32_t* const val[2], uint64_t n, int lo, int passes, bool iota,
                     uint32_t* hist, uint8_t* status, uint32_t* d_err, int& cur, cudaStream_t s,
                     const uint32_t* skip = nullptr) {
  if (n == 0 || passes == 0) return WTG_OK;
  const uint64_t hist_bytes = (uint64_t)passes * RS_RADIX * sizeof(uint32_t), status_bytes = radix_status_bytes(n, passes);
  if ((uint8_t*)hist + hist_bytes == status) {
    WTG_CK(cudaMemsetAsync(hist, 0, hist_bytes + status_bytes, s));
  } else {
    WTG_CK(cudaMemsetAsync(hist, 0, hist_bytes, s));
    WTG_CK(cudaMemsetAsync(status, 0, status_bytes, s));
  }
  const uint64_t blocks = (n + 8 * RS_THREADS - 1) / (8 * RS_THREADS);
  radix_hist_kernel<K><<<(unsigned)(blocks < 152 * 8 ? blocks : 152 * 8), RS_THREADS, 0, s>>>(key[cur], n, lo, passes,
                                                                                             hist, skip);
  count_launch();
  WTG_CK(cudaGetLastError());
  radix_bases_kernel<<<passes, RS_RADIX, 0, s>>>(hist);
  count_launch();
  WTG_CK(cudaGetLastError());
  return n < (1ull << 30) ? radix_passes<K, uint32_t>(key, val, n, lo, passes, iota, hist, status, d_err, cur, s, skip)
                          : radix_passes<K, uint64_t>(key, val, n, lo, passes, iota, hist, status, d_err, cur, s,
                                                      skip);
}

}  // namespace wtg
