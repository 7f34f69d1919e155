// wtg_pass_last.cu -- count and node passes, and the pass of a tree's last
// group of levels (bits only).
#include <algorithm>

#include "wtg_pass.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(build)

int lv_sm_count() {
  static const int n = [] {
    int dev = 0, k = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&k, cudaDevAttrMultiProcessorCount, dev);
    return k > 0 ? k : 1;
  }();
  return n;
}

int count_cpw(uint64_t nchunks) {
  const uint64_t c = nchunks / ((uint64_t)LV_WARPS * lv_sm_count() * 8);
  return c >= 8 ? 8 : c >= 4 ? 4 : c >= 2 ? 2 : 1;
}

namespace {

template <typename T, int TB>
int count_t(const LevelGroup& a, uint32_t tile0, uint32_t tile1, cudaStream_t s) {
  static int per_sm = 0;
  const PassArgs& p = a.pass;
  return launch_resident(count_kernel<T, TB>, per_sm, tile1 - tile0, 0, s, p.src, p.n, p.ds + a.tau - TB,
                         p.nchunks, a.cpw, a.chunkpre, a.status, a.sstride, a.counter, tile0, tile1, p.err, p.huff);
}

template <typename T, int TB>
int nodes_t(const LevelGroup& a, cudaStream_t s) {
  static int per_sm = 0;
  const PassArgs& p = a.pass;
  const uint64_t ctas = std::max(((uint64_t)p.nodes + LV_WARPS - 1) / LV_WARPS,
                                 p.nodes > 1 ? ((uint64_t)p.nchunks + LV_THREADS - 1) / LV_THREADS : 1);
  return launch_resident(node_pass_kernel<T, TB>, per_sm, ctas, 0, s, (const T*)p.src, p.n, p.ds + a.tau - TB, p.level,
                         a.C, a.Z, p.chunkpre, p.nchunks, (int)a.scatter, a.rec, a.cnode);
}

template <typename T, int TAU>
int last_t(const LevelGroup& a, cudaStream_t s) {
  static int per_sm = 0;
  const PassArgs& p = a.pass;
  const uint64_t ctas = ((uint64_t)p.nchunks + LV_WARPS - 1) / LV_WARPS;
  if constexpr (TAU == 1) {
    return launch_resident(single_level_kernel<T>, per_sm, ctas, 0, s, (const T*)p.src, p.n, p.ds, p.level, p.nchunks,
                           p.bits);
  } else {
    return launch_resident(level_pass_kernel<T, T, TAU, false, (sizeof(T) == 4 ? 2 : 3)>, per_sm, ctas,
                           lv_smem<T, false>(), s, p);
  }
}

}  // namespace

#define WTG_BY_BYTES(b, f, ...)               \
  switch (b) {                                \
    case 1: return f(uint8_t, __VA_ARGS__);   \
    case 2: return f(uint16_t, __VA_ARGS__);  \
    default: return f(uint32_t, __VA_ARGS__); \
  }

int launch_count(const LevelGroup& a, uint32_t tile0, uint32_t tile1, cudaStream_t s) {
  if (tile1 <= tile0) return WTG_OK;
#define WTG_F(T, TB) count_t<T, TB>(a, tile0, tile1, s)
  switch (a.scatter ? 4 : a.tau - 1) {
    case 1: WTG_BY_BYTES(a.src_bytes, WTG_F, 1)
    case 2: WTG_BY_BYTES(a.src_bytes, WTG_F, 2)
    case 3: WTG_BY_BYTES(a.src_bytes, WTG_F, 3)
    default: WTG_BY_BYTES(a.src_bytes, WTG_F, 4)
  }
#undef WTG_F
}

int launch_nodes(const LevelGroup& a, cudaStream_t s) {
#define WTG_F(T, TB) nodes_t<T, TB>(a, s)
  switch (a.scatter ? 4 : a.tau - 1) {
    case 1: WTG_BY_BYTES(a.src_bytes, WTG_F, 1)
    case 2: WTG_BY_BYTES(a.src_bytes, WTG_F, 2)
    case 3: WTG_BY_BYTES(a.src_bytes, WTG_F, 3)
    default: WTG_BY_BYTES(a.src_bytes, WTG_F, 4)
  }
#undef WTG_F
}

int launch_pass(const LevelGroup& a, cudaStream_t s) {
  if (a.scatter) return launch_pass_scatter(a, s);
#define WTG_F(T, TAU) last_t<T, TAU>(a, s)
  switch (a.tau) {
    case 1: WTG_BY_BYTES(a.src_bytes, WTG_F, 1)
    case 2: WTG_BY_BYTES(a.src_bytes, WTG_F, 2)
    case 3: WTG_BY_BYTES(a.src_bytes, WTG_F, 3)
    default: WTG_BY_BYTES(a.src_bytes, WTG_F, 4)
  }
#undef WTG_F
}

}  // namespace wtg
