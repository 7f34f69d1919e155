// wtg_pass_scatter.cu -- the pass of a group of four levels that another
// group follows: bits and scatter.
#include "wtg_pass.cuh"

namespace wtg {

namespace {

template <typename Tin, typename Tout>
int scatter_t(const LevelGroup& a, cudaStream_t s) {
  static int per_sm = 0;
  const uint64_t ctas = ((uint64_t)a.pass.nchunks + LV_WARPS - 1) / LV_WARPS;
  return launch_resident(level_pass_kernel<Tin, Tout, 4, true, (sizeof(Tin) == 4 ? 2 : 3)>, per_sm, ctas,
                         lv_smem<Tin, true>(), s, a.pass);
}

}  // namespace

int launch_pass_scatter(const LevelGroup& a, cudaStream_t s) {
  switch (a.src_bytes * 8 + a.dst_bytes) {
    case 4 * 8 + 4: return scatter_t<uint32_t, uint32_t>(a, s);
    case 4 * 8 + 2: return scatter_t<uint32_t, uint16_t>(a, s);
    case 4 * 8 + 1: return scatter_t<uint32_t, uint8_t>(a, s);
    case 2 * 8 + 2: return scatter_t<uint16_t, uint16_t>(a, s);
    case 2 * 8 + 1: return scatter_t<uint16_t, uint8_t>(a, s);
    default: return scatter_t<uint8_t, uint8_t>(a, s);
  }
}

}  // namespace wtg
