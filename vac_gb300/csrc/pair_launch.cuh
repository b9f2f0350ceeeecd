// pair_launch.cuh - launch of one instance of the pair sweep (sweep_pair.cu,
// roe_pair.cu).
#pragma once
#include "batch_items.cuh"
#include "sweep_pair.cuh"

namespace vacgpu {

template <int D, bool MHD, int LIMC, bool GEN, bool ROE>
static void launch_pair_one(const CUtensorMap* map, const FusedArgs& a, dim3 grid,
                            cudaStream_t st) {
  constexpr int NW = MHD ? 8 : 5;
  const int smem = pair_smem_floats(NW) * 4;
  auto k = k_sweep_pair<D, MHD, LIMC, GEN, ROE>;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = true;
  }
  k<<<grid, PT_NT, smem, st>>>(*map, a);
}

template <int D, bool MHD, int LIMC, bool ROE>
static void launch_pair_gen(const CUtensorMap* map, const FusedArgs& a, dim3 grid,
                            cudaStream_t st) {
  if (pair_general(a, MHD))
    launch_pair_one<D, MHD, LIMC, true, ROE>(map, a, grid, st);
  else
    launch_pair_one<D, MHD, LIMC, false, ROE>(map, a, grid, st);
}

// The Roe instances (MHD, woodward or minmod): false where there is none.
bool launch_pair_roe(const FusedArgs& a, int D, const CUtensorMap* map, dim3 grid,
                     cudaStream_t st);

}  // namespace vacgpu
