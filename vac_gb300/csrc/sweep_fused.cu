// sweep_fused.cu - instances and launcher of the fused mixed-precision sweep.
#include <cstdlib>
#include <cstring>

#include "sweep_fused.cuh"

namespace vacgpu {

int fused_smem_bytes(int nw, int k) { return fused_smem_floats(nw, k) * 4; }

bool launch_sweep_pair(FusedArgs a, int D, bool mhd, const void* tmap, int nzc,
                       cudaStream_t st);
bool launch_sweep_line2(const FusedArgs& a, const float* win, int D, bool mhd,
                        cudaStream_t st);

template <int NDIM, int D, bool MHD, int LIMC, int PMF>
static void launch_pmf(const CUtensorMap* map, const FusedArgs& a, dim3 grid,
                       cudaStream_t st) {
  constexpr int NW = MHD ? 2 + 2 * NDIM : 2 + NDIM;
  const int smem = fused_smem_floats(NW, fused_kind(NDIM, D)) * 4;
  auto k = k_sweep_fused<NDIM, D, MHD, PREC_FF, LIMC, PMF>;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = true;
  }
  k<<<grid, FT_NT, smem, st>>>(*map, a);
}

// VACGPU_FLUX_PRESSURE=f32: FP32 pressure recovery in the fluxes (the wave
// speeds keep the double-float recovery).  Read once per process.
static bool flux_pressure_f32() {
  static const bool f = [] {
    const char* e = getenv("VACGPU_FLUX_PRESSURE");
    return e && !strcmp(e, "f32");
  }();
  return f;
}

template <int NDIM, int D, bool MHD, int LIMC>
static void launch_lim(const CUtensorMap* map, const FusedArgs& a, dim3 grid,
                       cudaStream_t st) {
  if (flux_pressure_f32())
    launch_pmf<NDIM, D, MHD, LIMC, PREC_F32>(map, a, grid, st);
  else
    launch_pmf<NDIM, D, MHD, LIMC, PREC_FF>(map, a, grid, st);
}

template <int NDIM, int D, bool MHD>
static void launch_one(const CUtensorMap* map, const FusedArgs& a, dim3 grid,
                       cudaStream_t st) {
  constexpr int NW = MHD ? 2 + 2 * NDIM : 2 + NDIM;
  int l0 = a.ph.lim[0];
  bool uniform = a.ph.typefull != VACGPU_TVDLF1;
  for (int v = 1; v < NW; v++) uniform = uniform && a.ph.lim[v] == l0;
  if (uniform && l0 == VACGPU_LIM_WOODWARD)
    launch_lim<NDIM, D, MHD, LIMC_WOODWARD>(map, a, grid, st);
  else if (uniform && l0 == VACGPU_LIM_MINMOD)
    launch_lim<NDIM, D, MHD, LIMC_MINMOD>(map, a, grid, st);
  else
    launch_lim<NDIM, D, MHD, LIMC_RUNTIME>(map, a, grid, st);
}

bool pair_applies(const FusedArgs& a, bool mhd);
bool pair_general(const FusedArgs& a, bool mhd);
bool line2_applies(const FusedArgs& a, bool mhd);

// The fused sweeps with the Roe dissipation of 'tvdmu': ideal MHD without an
// entropy fix (the fixes modify the normalised eigenvalues, which the split
// kernels keep), on the grids of the two-cells-per-thread kernels alone.
// (HD stays on the split kernels, whose average is in double.)
bool fused_roe_applies(const DevGrid& g, const DevPhys& ph, int ndir, bool mhd) {
  if (ph.typefull != VACGPU_TVDMU || !mhd || ndir != g.ndim) return false;
  for (int il = 0; il < 2 + 2 * ndir; il++)
    if (ph.typeentropy[il] != VACGPU_ENTROPY_NUL) return false;
  FusedArgs a;
  memset(&a, 0, sizeof(a));
  a.g = g;
  a.ph = ph;
  return g.ndim == 3 ? pair_applies(a, mhd) : g.ndim == 2 && line2_applies(a, mhd);
}

// Planes per CTA (z chunk) of the one-cell kernel over `tiles` column tiles
// and n planes where the caller fixes none, as pair_chunk (sweep_pair.cu): the
// longest that gives so many waves of two CTAs per SM, else the longest of at
// most 8 that gives 250 CTAs, down to 2.  us a sweep by planes per CTA, the
// rule's choice first (MHD vanleer periodic; superbee with outflow faces; gas,
// vanleer with outflow faces):
//   64^3         35 (4; 8: 44, 32: 126)    46 (59, 175)       32 (40, 112)
//   128^3       165 (8; 12: 160, 32: 187) 200 (193, 246)     116 (111, 149)
//   130x127x133 177 (12; 16: 194, 32: 239) 218 (230, 299)    127 (129, 172)
//   192^3       437 (16-24; 12: 440, 32: 438) 520 (518, 549) 284 (282, 304)
//   256^3       921 (24; 48: 914, 32: 929) 1052 (1068, 1084) 550 (577, 576)
//   320x300x310 1538 (48; 24: 1584, 32: 1560) 1743 (1782, 1757)
// A trial in a grid's first call, before 32 planes were taken for every grid,
// found 169, 194, 437, 916 and 1544 (207, 231, 517, 1056 and 1748) from 128^3 on.
static int fused_chunk(int tiles, int n) {
  static const struct {
    int z, waves;
  } longer[] = {{48, 8}, {24, 4}, {16, 5}, {12, 3}};
  auto ctas = [&](int z) { return (long long)tiles * ((n + z - 1) / z); };
  for (const auto& l : longer)
    if (ctas(l.z) >= l.waves * 2 * NUM_SMS) return l.z;
  for (int z : {8, 6, 4, 3})
    if (ctas(z) >= 250) return z;
  return 2;
}

bool launch_sweep_fused(const SweepArgs& s, const void* tmap, const float* win, float* wout,
                        const float* const* idxf, int nzc, cudaStream_t st) {
  const int nd = s.g.ndim;
  if (s.d0 != s.d1 || s.ndir != nd || (nd != 2 && nd != 3)) return false;
  for (int d = 0; d < nd; d++)
    if (s.ph.gmap[d][0] == GMAP_MIXED || s.ph.gmap[d][1] == GMAP_MIXED)
      return false;
  FusedArgs a;
  memset(&a, 0, sizeof(a));
  a.g = s.g;
  a.ph = s.ph;
  for (int d = 0; d < 3; d++) {
    a.dxf[d] = s.a.dxf[d];
    a.idxf[d] = idxf[d];
  }
  a.ctrl = s.ctrl;
  a.wout = wout;
  for (int d = 0; d < 3; d++) a.gravf[d] = (float)s.ph.src_par[d];
  a.cfl = s.ph.courantpar > 0.0;
  const int nw = s.mhd ? 2 + 2 * s.ndir : 2 + s.ndir;
  for (int d = 0; d < 3; d++)
    for (int v = 0; v < nw; v++) {
      if (s.ph.typeB[2 * d][v] == VACGPU_BC_PERIODIC) a.periodic_mask[d] |= 1 << v;
      if (s.ph.typeB[2 * d][v] == VACGPU_BC_ASYMM) a.asymm_lo[d] |= 1 << v;
      if (s.ph.typeB[2 * d + 1][v] == VACGPU_BC_ASYMM) a.asymm_hi[d] |= 1 << v;
    }
  // 3-D grids: the two-cells-per-thread kernel (packed FP32) where it
  // applies; VACGPU_PAIR=0 keeps the one-cell kernel
  if (nd == 3 && launch_sweep_pair(a, s.d0, s.mhd, tmap, nzc, st)) {
    if (pair_general(a, s.mhd)) launch_ghost_yz_mixed(s, wout, st);
    return true;
  }
  // 2-D grids: the warp-marching two-cells-per-thread kernel where it applies
  if (nd == 2 && launch_sweep_line2(a, win, s.d0, s.mhd, st)) return true;
  // the one-cell kernel: tiles over x and the row axis, z chunks along the
  // marching axis
  const int kind = fused_kind(nd, s.d0);
  const int tx = kind == 0 ? TileCfg<0>::TX : TileCfg<1>::TX;
  const int ty = kind == 1 ? TileCfg<1>::TY : TileCfg<0>::TY;
  const int ar = kind == 2 && s.d0 == 1 ? 2 : 1;
  const int am = kind == 2 ? s.d0 : 2;
  const int nxt = (s.g.nx[0] + tx - 1) / tx, nyt = (s.g.nx[ar] + ty - 1) / ty;
  if (nzc <= 0) nzc = nd == 3 ? fused_chunk(nxt * nyt, s.g.nx[am]) : 1;
  a.nzc = nzc;
  dim3 grid(nxt, nyt, nd == 3 ? (s.g.nx[am] + nzc - 1) / nzc : 1);
  const CUtensorMap* map = (const CUtensorMap*)tmap;
  const int D = s.d0;
#define L1(ND, DD)                                              \
  if (nd == ND && D == DD) {                                    \
    if (s.mhd)                                                  \
      launch_one<ND, DD, true>(map, a, grid, st);               \
    else                                                        \
      launch_one<ND, DD, false>(map, a, grid, st);              \
    return true;                                                \
  }
  L1(2, 0) L1(2, 1) L1(3, 0) L1(3, 1) L1(3, 2)
#undef L1
  return false;
}

}  // namespace vacgpu
