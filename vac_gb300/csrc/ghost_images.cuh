// ghost_images.cuh - getboundary's ghost fill done by the cells it copies
// from: a kernel that writes a new cell value also writes it to every ghost
// position whose boundary maps land on that cell (the region-by-region
// copies of src/vacgrid.t:195-413 composed), so no launch has to fill ghost
// cells after it.  For grids whose faces have one index map for every
// variable (gmap not GMAP_MIXED), periodic faces in pairs and at least four
// cells a dimension.
#pragma once
#include "vacgpu_internal.h"

namespace vacgpu {

// Ghost-cell preimages of the mesh index gi along dimension d (n cells,
// ghost-range indices 0..n+3, n >= 4): up to two ghost positions p1, p2
// whose boundary map lands on gi, and the 'asymm' sign mask of the first.
// periodic: gi-n for gi >= n, gi+n for gi < 4; cont: 0 and 1 for gi = 2,
// n+2 and n+3 for gi = n+1; symm/asymm: 3-gi for gi < 4, 2n+3-gi for
// gi >= n (negated for 'asymm' variables).
__device__ __forceinline__ int ghost_preimages(const DevGrid& g, const DevPhys& ph, int d, int gi,
                                               int& p1, int& f1, int& p2) {
  const int n = g.nx[d];
  const int mlo = ph.gmap[d][0], mhi = ph.gmap[d][1];
  p1 = p2 = gi;
  f1 = 0;
  if (gi < 4) {
    if (mlo == GMAP_CONT && gi == 2) {
      p1 = 0;
      p2 = 1;
      return 2;
    }
    if (mlo == GMAP_MIRROR) {
      p1 = 3 - gi;
      f1 = ph.asym[d][0];
      return 1;
    }
    if (mhi == GMAP_PERIODIC) {
      p1 = gi + n;
      return 1;
    }
  }
  if (gi >= n) {
    if (mhi == GMAP_CONT && gi == n + 1) {
      p1 = n + 2;
      p2 = n + 3;
      return 2;
    }
    if (mhi == GMAP_MIRROR) {
      p1 = 2 * n + 3 - gi;
      f1 = ph.asym[d][1];
      return 1;
    }
    if (mlo == GMAP_PERIODIC) {
      p1 = gi - n;
      return 1;
    }
  }
  return 0;
}

// The ghost images of the cell gc (ghost-range coordinates, element offset
// off) with values s: the positions whose coordinates are gc's own or
// preimages in every dimension, at least one of them a preimage.
template <int NDIM, int NW, typename T, typename R>
__device__ __forceinline__ void write_ghost_images(const DevGrid& g, const DevPhys& ph,
                                                   T* __restrict__ w, const int* gc,
                                                   long long off, const R* s) {
  int x1, x2, fx, y1 = 0, y2 = 0, fy = 0, z1 = 0, z2 = 0, fz = 0;
  const int nx_ = 1 + ghost_preimages(g, ph, 0, gc[0], x1, fx, x2);
  const int ny_ = NDIM > 1 ? 1 + ghost_preimages(g, ph, 1, gc[1], y1, fy, y2) : 1;
  const int nz_ = NDIM > 2 ? 1 + ghost_preimages(g, ph, 2, gc[2], z1, fz, z2) : 1;
#pragma unroll 1
  for (int k = 0; k < nz_; k++) {
    const int pz = k == 0 ? gc[2] : (k == 1 ? z1 : z2);
    const int sz = k == 1 ? fz : 0;
#pragma unroll 1
    for (int j = 0; j < ny_; j++) {
      const int py = j == 0 ? gc[1] : (j == 1 ? y1 : y2);
      const int sy = j == 1 ? fy : 0;
      const long long orow =
          off + (long long)(pz - gc[2]) * g.plane + (long long)(py - gc[1]) * g.P;
#pragma unroll 1
      for (int i = 0; i < nx_; i++) {
        if ((i | j | k) == 0) continue;
        const int px = i == 0 ? gc[0] : (i == 1 ? x1 : x2);
        const int fl = (i == 1 ? fx : 0) ^ sy ^ sz;
        const long long o = orow + (px - gc[0]);
#pragma unroll
        for (int v = 0; v < NW; v++) w[o + v * g.vs] = ((fl >> v) & 1) ? T(-s[v]) : T(s[v]);
      }
    }
  }
}

// The grid's faces admit ghost images.
inline bool ghost_images_apply(const DevGrid& g, const DevPhys& ph) {
  for (int d = 0; d < g.ndim; d++)
    if (ph.gmap[d][0] == GMAP_MIXED || ph.gmap[d][1] == GMAP_MIXED || g.nx[d] < 4 ||
        (ph.gmap[d][0] == GMAP_PERIODIC) != (ph.gmap[d][1] == GMAP_PERIODIC))
      return false;
  return true;
}

}  // namespace vacgpu
