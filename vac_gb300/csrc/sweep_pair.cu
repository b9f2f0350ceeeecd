// sweep_pair.cu - instances and launcher of the two-cells-per-thread fused
// sweep of 3-D grids (mixed precision).
#include <cstdlib>
#include <cstring>

#include "batch_items.cuh"
#include "pair_launch.cuh"

namespace vacgpu {

// The grid needs the general form of the pair sweep (PairSweep's GEN):
// gravity, a non-periodic face, split sources, no Powell terms for MHD, or
// no CFL maximum.
bool pair_general(const FusedArgs& a, bool mhd) {
  const int all = (1 << (mhd ? 8 : 5)) - 1;
  bool gen = a.ph.src_id != VACGPU_SRC_NONE || !a.ph.sourceunsplit || !a.cfl ||
             (mhd && !a.ph.divbfix);
  for (int d = 0; d < 3; d++) gen = gen || a.periodic_mask[d] != all;
  return gen;
}

// VACGPU_PAIR=0 keeps the one-cell kernel for every grid (read once)
bool pair_enabled() {
  static const bool on = [] {
    const char* e = getenv("VACGPU_PAIR");
    return !(e && atoi(e) == 0);
  }();
  return on;
}

// The pair sweep runs 3-D sweeps with one limiter for every variable
// (minmod or woodward).
bool pair_applies(const FusedArgs& a, bool mhd) {
  if (!pair_enabled()) return false;
  const int nw = mhd ? 8 : 5;
  const int l0 = a.ph.lim[0];
  bool uniform = a.ph.typefull != VACGPU_TVDLF1;
  for (int v = 1; v < nw; v++) uniform = uniform && a.ph.lim[v] == l0;
  if (!uniform || (l0 != VACGPU_LIM_WOODWARD && l0 != VACGPU_LIM_MINMOD)) return false;
  // the pairs' 8-byte shared and global accesses need an even first column
  // (state rows start at xpad, a multiple of 32 minus 2 for FP32 states)
  return a.g.ndim == 3 && !(a.g.xpad & 1) && !(a.g.P & 1);
}

// Planes per CTA (z chunk) of a sweep over `tiles` column tiles and n planes
// where the caller fixes none: the longest of 24, 20, 16 and 12 planes that
// gives at least three waves of three CTAs per SM, else the longest of at most
// 8 that gives 350 CTAs, down to 2.  Every chunk predicts two planes beyond
// its own, but the march of one CTA is a serial chain (1.9 us a plane alone on
// its SM, 2.8 beside two others), so a small grid wants many short ones, and a
// large one enough of them that the last wave leaves few slots idle.  The
// thresholds come from the TVDLF MHD kernel; Roe's, which runs two CTAs per
// SM, and gas's want nearly the same chunks.  us a sweep of periodic grids by
// planes per CTA, the rule's choice first:
//   MHD  64^3 26.6 (3-4; 8: 33, 32: 88)      128x113x120 86 (8; 16: 88, 32: 108)
//       192^3 240 (20; 8: 254, 64: 283)           256^3 513 (24; 12: 525, 64: 558)
//   Roe  64^3 31.8 (3-4; 4: 29, 32: 83)      128x113x120 99.6 (8; 16: 98, 32: 110)
//       192^3 295 (20; 8: 316, 32: 305)           256^3 639 (24; 12: 661, 32: 649)
//   gas  64^3 17.0 (3-4; 8: 20, 32: 50)      128x113x120 46.6 (8; 16: 46, 32: 61)
//       192^3 128 (20; 8: 133, 64: 145)           256^3 263 (24; 12: 267, 64: 297)
// With outflow faces likewise; over 48^3 to 320x300x310 no other chunk was
// faster by more than 3 % for MHD and gas, or 2 % for Roe but for the 64^3
// above.  (A trial of each chunk in a grid's first call, before, cost that
// call six steps and gained nothing.)
static int pair_chunk(int tiles, int n) {
  for (int z : {24, 20, 16, 12})
    if ((long long)tiles * ((n + z - 1) / z) >= 3 * 3 * NUM_SMS) return z;
  for (int z : {8, 6, 4, 3})
    if ((long long)tiles * ((n + z - 1) / z) >= 350) return z;
  return 2;
}

// nzc <= 0: pair_chunk's choice.  False: not applicable, use the one-cell
// kernel.
bool launch_sweep_pair(FusedArgs a, int D, bool mhd, const void* tmap, int nzc,
                       cudaStream_t st) {
  if (!pair_applies(a, mhd)) return false;
  const int l0 = a.ph.lim[0];
  const int tx = D == 0 ? 30 : 32;
  const int ar = D == 1 ? 2 : 1, am = D == 0 ? 2 : D;
  const int nxt = D == 0 ? (a.g.nx[0] + 1 + tx - 1) / tx : (a.g.nx[0] + tx - 1) / tx;
  const int nyt = (a.g.nx[ar] + 7) / 8;
  if (nzc <= 0) nzc = pair_chunk(nxt * nyt, a.g.nx[am]);
  a.nzc = nzc;
  dim3 grid(nxt, nyt, (a.g.nx[am] + nzc - 1) / nzc);
  const CUtensorMap* map = (const CUtensorMap*)tmap;
  // the Roe instances are a unit of their own (roe_pair.cu)
  if (a.ph.typefull == VACGPU_TVDMU) return launch_pair_roe(a, D, map, grid, st);
#define LP(DD, M, L) launch_pair_gen<DD, M, L, false>(map, a, grid, st)
#define LPD(DD)                                                              \
  if (D == DD) {                                                             \
    if (mhd) {                                                               \
      if (l0 == VACGPU_LIM_WOODWARD) LP(DD, true, LIMC_WOODWARD);            \
      else LP(DD, true, LIMC_MINMOD);                                        \
    } else {                                                                 \
      if (l0 == VACGPU_LIM_WOODWARD) LP(DD, false, LIMC_WOODWARD);           \
      else LP(DD, false, LIMC_MINMOD);                                       \
    }                                                                        \
    return true;                                                             \
  }
  LPD(0) LPD(1) LPD(2)
#undef LPD
#undef LP
  return false;
}

// ------------------------------------------------------- batched grids

// The pair sweep over a batch work list: each CTA takes items
// blockIdx.x, blockIdx.x + gridDim.x, ... in turn, with the item's grid
// arguments copied to shared memory; the TMA barriers' phases carry over
// from item to item.
template <int D, bool MHD, int LIMC, bool GEN>
__global__ void __launch_bounds__(PT_NT, 3)
    kb_sweep_pair(const BItem* __restrict__ items, int nitems,
                  const BInst* __restrict__ insts, const CUtensorMap* maps, int sweep) {
  extern __shared__ __align__(128) float dsm[];
  __shared__ __align__(8) unsigned long long bars[FWRING];
  __shared__ __align__(16) FusedArgs fa;
  __shared__ int mapidx;
  init_bars(bars);
  int uses[FWRING] = {0, 0, 0, 0};
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const BItem item = items[it];
    const BInst* in = insts + item.inst;
    {
      const int* src = (const int*)&in->fa;
      int* dst = (int*)&fa;
      for (int k = threadIdx.x; k < (int)(sizeof(FusedArgs) / 4); k += blockDim.x)
        dst[k] = src[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int src = in->fa.ctrl->cur ^ (sweep & 1);
      fa.wout = in->buf[src ^ 1];
      mapidx = item.inst * 4 + src * 2 + (D == 1);
    }
    __syncthreads();
    const bool ok = PairSweep<D, MHD, LIMC, GEN>::run(&maps[mapidx], fa, dsm, item.bx, item.by,
                                                     item.bz, bars, uses, (unsigned)it);
    __syncthreads();
    if (!ok) return;
  }
}

template <int D, bool MHD, int LIMC, bool GEN>
static void launch_kb_pair(const BItem* items, int nitems, const BInst* insts,
                           const CUtensorMap* maps, int sweep, int ctas, cudaStream_t st) {
  constexpr int NW = MHD ? 8 : 5;
  const int smem = pair_smem_floats(NW) * 4;
  auto k = kb_sweep_pair<D, MHD, LIMC, GEN>;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = true;
  }
  k<<<ctas, PT_NT, smem, st>>>(items, nitems, insts, maps, sweep);
}

bool launch_batch_pair(const BItem* items, int nitems, const BInst* insts,
                       const CUtensorMap* maps, int sweep, int D, bool mhd, int lim,
                       bool gen, int ctas, cudaStream_t st) {
  if (ctas <= 0 || ctas > nitems) ctas = nitems;
#define KP(DD, M, L)                                                          \
  {                                                                           \
    if (gen)                                                                  \
      launch_kb_pair<DD, M, L, true>(items, nitems, insts, maps, sweep, ctas, st); \
    else                                                                      \
      launch_kb_pair<DD, M, L, false>(items, nitems, insts, maps, sweep, ctas, st); \
    return true;                                                              \
  }
#define KPD(DD)                                                               \
  if (D == DD) {                                                              \
    if (mhd) {                                                                \
      if (lim == VACGPU_LIM_WOODWARD) KP(DD, true, LIMC_WOODWARD)             \
      else KP(DD, true, LIMC_MINMOD)                                          \
    } else {                                                                  \
      if (lim == VACGPU_LIM_WOODWARD) KP(DD, false, LIMC_WOODWARD)            \
      else KP(DD, false, LIMC_MINMOD)                                         \
    }                                                                         \
  }
  KPD(0) KPD(1) KPD(2)
#undef KPD
#undef KP
  return false;
}

}  // namespace vacgpu
