// wtg_pass_huff.cu -- the passes of a group of four levels of a Huffman-shaped
// tree: bytes read through the group's digit table (see HuffGroup).
#include "wtg_pass.cuh"

namespace wtg {

WTG_WAIT_LIMIT_SETTER(huff_pass)

namespace {

template <int TB>
int count_t(const LevelGroup& a, uint32_t tiles, cudaStream_t s) {
  static int per_sm = 0;
  const PassArgs& p = a.pass;
  return launch_resident(count_kernel<uint16_t, TB, true>, per_sm, tiles, 0, s, p.src, p.n, p.ds + 4 - TB, p.nchunks,
                         a.cpw, a.chunkpre, a.status, a.sstride, a.counter, 0u, tiles, p.err, p.huff);
}

template <bool SCATTER>
int pass_t(const LevelGroup& a, cudaStream_t s) {
  static int per_sm = 0;
  const uint64_t ctas = ((uint64_t)a.pass.nchunks + LV_WARPS - 1) / LV_WARPS;
  return launch_resident(level_pass_kernel<uint16_t, uint8_t, 4, SCATTER, 3, true>, per_sm, ctas,
                         lv_smem<uint16_t, SCATTER>(), s, a.pass);
}

}  // namespace

int launch_huff_count(const LevelGroup& a, uint32_t tiles, cudaStream_t s) {
  return a.scatter ? count_t<4>(a, tiles, s) : count_t<3>(a, tiles, s);
}

int launch_huff_pass(const LevelGroup& a, cudaStream_t s) {
  return a.scatter ? pass_t<true>(a, s) : pass_t<false>(a, s);
}

}  // namespace wtg
