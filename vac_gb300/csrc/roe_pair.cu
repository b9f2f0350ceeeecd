// roe_pair.cu - the pair sweep's instances with the MHD Roe dissipation
// ('tvdmu' on the mixed path, 3-D).
#include "pair_launch.cuh"

namespace vacgpu {

bool launch_pair_roe(const FusedArgs& a, int D, const CUtensorMap* map, dim3 grid,
                     cudaStream_t st) {
  const int l0 = a.ph.lim[0];
#define LR(DD)                                                             \
  if (D == DD) {                                                           \
    if (l0 == VACGPU_LIM_WOODWARD)                                         \
      launch_pair_gen<DD, true, LIMC_WOODWARD, true>(map, a, grid, st);    \
    else                                                                   \
      launch_pair_gen<DD, true, LIMC_MINMOD, true>(map, a, grid, st);      \
    return true;                                                           \
  }
  LR(0) LR(1) LR(2)
#undef LR
  return false;
}

}  // namespace vacgpu
