// wtg_hist.cuh -- byte counts of a text (internal).
#pragma once
#include "wtg_internal.cuh"

namespace wtg {

// Byte counts.  Sixteen copies of a byte's counter, a lane's by its number,
// lie side by side, so that the lanes of a warp that read the same byte meet on
// few words: the shared atomics bound it, not the read (2^26 zipf bytes 20 us,
// 105 us with one copy a CTA; 2^27 DNA codes 35 us, 175
// with one a warp).
constexpr int HIST_COPIES = 16;
template <typename T>
__global__ void __launch_bounds__(512)
    byte_hist_kernel(const uint8_t* __restrict__ s, uint64_t n, T* __restrict__ hist) {
  __shared__ uint32_t h[256 * HIST_COPIES];
  for (uint32_t i = threadIdx.x; i < 256 * HIST_COPIES; i += blockDim.x) h[i] = 0;
  __syncthreads();
  uint32_t* const mine = h + (threadIdx.x & (HIST_COPIES - 1));
  const uint64_t head = min(n, (uint64_t)((16 - ((uintptr_t)s & 15)) & 15)), quads = (n - head) / 16;
  const uint4* __restrict__ q = reinterpret_cast<const uint4*>(s + head);
  const uint64_t me = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = me; i < quads; i += stride) {
    const uint4 v = __ldg(q + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 16; ++k) atomicAdd(mine + ((w[k / 4] >> (8 * (k % 4))) & 0xFFu) * HIST_COPIES, 1u);
  }
  const uint64_t rest = n - 16 * quads;  // below 32: the bytes before and after the 16-byte words
  if (me < rest) atomicAdd(mine + s[me < head ? me : 16 * quads + me] * HIST_COPIES, 1u);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) {
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < HIST_COPIES; ++k) sum += h[i * HIST_COPIES + ((k + i) & (HIST_COPIES - 1))];
    if (sum) atomicAdd(&hist[i], (T)sum);
  }
}

}  // namespace wtg
