// wtg_pass.cuh -- launchers of the level passes (internal; the kernels are in
// wtg_levels.cuh, instantiated by wtg_pass_scatter.cu, wtg_pass_last.cu and
// wtg_pass_huff.cu).
#pragma once
#include "wtg_levels.cuh"

namespace wtg {

// One group of tau <= 4 levels (all but a tree's last group: four, scattering).
struct LevelGroup {
  PassArgs pass;
  int tau;
  bool scatter;
  int src_bytes, dst_bytes;  // 1, 2 or 4 bytes a symbol; dst_bytes 0 without scatter
  uint32_t* C;               // node tables in heap order
  uint32_t* Z;
  uint32_t* chunkpre;
  uint32_t* cnode;
  uint32_t* rec;
  int cpw;                   // chunks per warp of a count tile
  uint32_t* counter;
  uint64_t* status;
  uint32_t sstride;
};

// digit counts of tiles [tile0, tile1) (in order, over one or several calls)
int launch_count(const LevelGroup& a, uint32_t tile0, uint32_t tile1, cudaStream_t s);
int launch_nodes(const LevelGroup& a, cudaStream_t s);
int launch_pass(const LevelGroup& a, cudaStream_t s);
int launch_pass_scatter(const LevelGroup& a, cudaStream_t s);
// the two passes of a Huffman-shaped tree's group (wtg_pass_huff.cu)
int launch_huff_count(const LevelGroup& a, uint32_t tiles, cudaStream_t s);
int launch_huff_pass(const LevelGroup& a, cudaStream_t s);

// chunks per warp of a count tile: more per tile (fewer look-backs) once the
// tiles still fill the chip eight times
int count_cpw(uint64_t nchunks);

int lv_sm_count();

// launches kernel K with as many CTAs as stay resident, at most `ctas`
template <typename F, typename... A>
int launch_resident(F kernel, int& per_sm, uint64_t ctas, size_t smem, cudaStream_t s, A... args) {
  if (!per_sm) {
    if (smem > 48 * 1024)
      WTG_CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int k = 0;
    WTG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, kernel, LV_THREADS, smem));
    per_sm = k > 0 ? k : 1;
  }
  const uint64_t most = (uint64_t)per_sm * lv_sm_count();
  kernel<<<(unsigned)(ctas < most ? ctas : most), LV_THREADS, smem, s>>>(args...);
  count_launch();
  WTG_CK(cudaGetLastError());
  return WTG_OK;
}

}  // namespace wtg
