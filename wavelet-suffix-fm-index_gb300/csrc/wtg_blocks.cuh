// wtg_blocks.cuh -- a bitvector's rank counts and bits in one 32-byte sector
// (internal): what large query batches probe instead of the rank_support_v
// table and the bitvector, whose entry and word are two sectors.
//
// Block b holds bits [192 b, 192 b + 192): {ones before it (32 bits, mod
// 2^32), ones of its first one and first two words (8 bits each), its three
// words}: 4/3 of the bits, where bits and rank table are 5/4.  Made per call
// from the two (a read and a write of the bitvector), so no state outlives
// the call and the reference layouts stay as they are.
#pragma once
#include "wtg_internal.cuh"

namespace wtg {

constexpr uint32_t BLOCK_BITS = 192;

inline uint64_t block_count(uint64_t size) { return size / BLOCK_BITS + 1; }  // position `size` has a block, too

struct BlockProbe {
  uint32_t ones;  // ones before the position (mod 2^32)
  uint32_t bit;   // the bit at it
};

// (kept out of L1: the probes of a batch hardly meet there, and the fills cost
// 10 % of the counting time)
__device__ __forceinline__ void block_load(const uint4* __restrict__ blocks, uint64_t b, uint64_t (&v)[4]) {
  asm volatile("ld.global.nc.L1::no_allocate.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
               : "l"(blocks + 2 * b));
}

__device__ __forceinline__ BlockProbe block_at(const uint64_t (&v)[4], uint32_t off) {
  const uint32_t w = off >> 6;
  const uint64_t word = w == 0 ? v[1] : w == 1 ? v[2] : v[3];
  const uint32_t sub = w ? (uint32_t)(v[0] >> (24 + 8 * w)) & 255u : 0u;
  BlockProbe r;
  r.ones = (uint32_t)v[0] + sub + __popcll(word & ((1ull << (off & 63)) - 1));
  r.bit = (uint32_t)(word >> (off & 63)) & 1u;
  return r;
}

// block and offset of a position
__device__ __forceinline__ uint64_t block_of(uint64_t pos, uint32_t& off) {
  const uint64_t w = pos >> 6;
  uint64_t b;
  if (w >> 32) b = w / 3;
  else b = __umulhi((uint32_t)w, 0xAAAAAAABu) >> 1;  // floor(w / 3), exact for 32 bits
  off = (uint32_t)(pos - b * BLOCK_BITS);
  return b;
}

static __global__ void __launch_bounds__(256)
    blocks_kernel(const uint64_t* __restrict__ words, const uint64_t* __restrict__ rt, uint64_t nwords, uint64_t count,
                  uint4* __restrict__ blocks, const uint32_t* __restrict__ wanted) {
  if (wanted && !*wanted) return;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < count; b += stride) {
    uint64_t w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = 3 * b + k < nwords ? __ldg(words + 3 * b + k) : 0ull;
    const uint64_t first = 3 * b;
    const uint64_t* e = rt + 2 * (first >> 3);
    const uint32_t k = (uint32_t)first & 7;
    const uint32_t ones = (uint32_t)__ldg(e) + (k ? (uint32_t)(__ldg(e + 1) >> (63 - 9 * k)) & 0x1FFu : 0u);
    const uint32_t c1 = __popcll(w[0]), c2 = c1 + __popcll(w[1]);
    uint64_t* o = reinterpret_cast<uint64_t*>(blocks + 2 * b);
    const uint64_t head = (uint64_t)ones | ((uint64_t)c1 << 32) | ((uint64_t)c2 << 40);
    *reinterpret_cast<ulonglong2*>(o) = make_ulonglong2(head, w[0]);
    *reinterpret_cast<ulonglong2*>(o + 2) = make_ulonglong2(w[1], w[2]);
  }
}

// Fills the blocks of a bitvector of `size` bits; wanted: a device word, and
// nothing is done where it is 0 (the grid is bounded so that this takes no time).
inline bool fill_blocks(uint4* blocks, const uint64_t* words, const uint64_t* rt, uint64_t size,
                        const uint32_t* wanted, cudaStream_t s) {
  const uint64_t count = block_count(size), ctas = (count + 255) / 256;
  blocks_kernel<<<(unsigned)(ctas < 152 * 64 ? ctas : 152 * 64), 256, 0, s>>>(words, rt, (size + 63) / 64, count, blocks,
                                                                            wanted);
  count_launch();
  return cudaGetLastError() == cudaSuccess;
}

// Blocks that a bitvector of `size` bits has, 0 where L1 holds it with its rank
// table (the blocks are read past it: 2^20 patterns of 100 symbols over 2^16
// symbols x 2 levels 1.1 ms, by blocks 2.2).
inline uint64_t blocks_in_reach(uint64_t size) { return size / 8 > (128u << 10) ? block_count(size) : 0; }

}  // namespace wtg
