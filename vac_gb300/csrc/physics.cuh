// physics.cuh - pointwise ideal-MHD / gamma-law HD physics of VAC 4.52 for
// the device, on one state vector u[NW] (conservative variables).
//
// The FP64 functions keep every Fortran array statement of the reference as
// the same sequence of IEEE operations (this header is compiled without FMA
// contraction for the FP64 path), so each value is bit-identical to the CPU
// restatement.  A factor that is a power of two is folded into an FMA where
// the reference multiplies by it and adds: the product is exact, so the
// FMA rounds once, where the reference's sum does, and the FP64 pipe, which
// bounds these kernels, issues one operation less.  A half is not exact in
// the subnormal range, which the fluxes and div B reach ahead of a front that
// spreads into gas at rest (half_plus); the pressure and the fast speed halve
// and quarter terms that are added to others of ordinary size.  Variable
// layout (src/vacpar.t.mhd:9-26, src/vacpar.t.hd:9-26):
//   rho=0, m_c=c (c=1..NDIR), e=NDIR+1, b_c=NDIR+1+c.
#pragma once
#include <cuda_runtime.h>

#include "vacgpu_internal.h"

namespace vacgpu {

template <int NDIR, bool MHD>
struct Lay {
  static constexpr int NW = MHD ? 2 + 2 * NDIR : 2 + NDIR;
  static constexpr int RHO = 0;
  static constexpr int M0 = 0;
  static constexpr int E = NDIR + 1;
  static constexpr int B0 = NDIR + 1;
};

// Constant sub-expressions of gamma live in DevPhys, evaluated once on the
// host in FP64 with the same operations the reference applies (so they are
// the same bits): pt1 = one-half*gamma, gm1 = gamma-one,
// pt3 = half*(gamma-one).
typedef DevPhys PhysConst;

// ------------------------------------------------------------------ FP64

// Several IEEE quotients by one denominator.  A state is divided by its
// density five times in a flux, and CUDA's division costs nine operations of
// the FP64 pipe each time; here the reciprocal is formed once and a quotient
// takes four: with y = RN(1/b) and yl = 1/b - y to a few bits,
// q = RN(a*y + RN(a*yl)) is within an ulp of a/b, its remainder r = a - b*q
// is exact, and RN(q + r*y) is then a/b correctly rounded (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34 (1990), theorem on quotients).  That holds
// away from overflow and underflow: b in [2^-100, 2^100] and |a| in
// [2^-800, 2^800], tested on the exponents.  A zero a over such a b is the
// quotient itself -- gas at rest or unmagnetised has one in most divisions,
// and CUDA's division leaves its fast path for it; everything else takes
// CUDA's division.
static __device__ __noinline__ double div_any(double a, double b) { return a / b; }
struct Rcp64 {
  double b, y, yl;
  bool ok;
};
__device__ __forceinline__ bool exponent_within(double x, unsigned e) {
  return (((unsigned)__double2hiint(x) >> 20 & 0x7ffu) - (1023u - e)) <= 2u * e;
}
__device__ __forceinline__ Rcp64 rcp64(double b) {
  Rcp64 r;
  r.b = b;
  r.y = __drcp_rn(b);
  r.yl = fma(-b, r.y, 1.0) * r.y;
  r.ok = __double2hiint(b) > 0 && exponent_within(b, 100);
  return r;
}
__device__ __forceinline__ double div64(double a, const Rcp64& r) {
  double q = fma(a, r.y, a * r.yl);
  q = fma(fma(-r.b, q, a), r.y, q);
  if (!(r.ok && exponent_within(a, 800)))
    q = r.ok && (__double_as_longlong(a) << 1) == 0 ? a : div_any(a, r.b);
  return q;
}

// 0.5*s may round: s is not zero and its half is subnormal
__device__ __forceinline__ bool half_rounds(double s) {
  const unsigned hi = (unsigned)__double2hiint(s) << 1;
  return hi < 0x00400000u && (hi | (unsigned)__double2loint(s)) != 0;
}
// 0.5*s + d with the product rounded first, as the reference has it
static __device__ __noinline__ double half_plus_any(double s, double d) { return 0.5 * s + d; }
__device__ __forceinline__ double half_plus(double s, double d) {
  return half_rounds(s) ? half_plus_any(s, d) : fma(0.5, s, d);
}

// getptotal, src/vacphys0.t.mhd:225-257 (unclipped total pressure)
template <int NDIR>
__device__ __forceinline__ double ptotal_mhd(const double* u, const Rcp64& ir,
                                             const PhysConst& k) {
  typedef Lay<NDIR, true> L;
  double bb = u[L::B0 + 1] * u[L::B0 + 1];
#pragma unroll
  for (int c = 2; c <= NDIR; c++) bb = bb + u[L::B0 + c] * u[L::B0 + c];
  double p = k.pt1 * bb;
  p = p + k.gm1 * u[L::E];
  double mm = u[1] * u[1];
#pragma unroll
  for (int c = 2; c <= NDIR; c++) mm = mm + u[c] * u[c];
  p = p - div64(k.pt3 * mm, ir);
  return p;
}

// getpthermal, src/vacphys0.t.mhd:165-222 (before clipping)
// (ir: u[0] and its reciprocal)
template <int NDIR>
__device__ __forceinline__ double pthermal_mhd_raw(const double* u, const Rcp64& ir,
                                                   const PhysConst& k) {
  typedef Lay<NDIR, true> L;
  double mm = u[1] * u[1];
#pragma unroll
  for (int c = 2; c <= NDIR; c++) mm = mm + u[c] * u[c];
  double p = div64(mm, ir);
#pragma unroll
  for (int c = 1; c <= NDIR; c++) p = p + u[L::B0 + c] * u[L::B0 + c];
  return k.gm1 * fma(-0.5, p, u[L::E]);  // e - 0.5*p
}

// getpthermal, src/vacphys0.t.hd:103-134 (before clipping)
template <int NDIR>
__device__ __forceinline__ double pthermal_hd_raw(const double* u, const Rcp64& ir,
                                                  const PhysConst& k) {
  typedef Lay<NDIR, false> L;
  double mm = u[1] * u[1];
#pragma unroll
  for (int c = 2; c <= NDIR; c++) mm = mm + u[c] * u[c];
  return k.gm1 * fma(-0.5, div64(mm, ir), u[L::E]);  // e - 0.5*mm/rho
}

__device__ __forceinline__ double clip_p(double p, double smallp) {
  return (p >= smallp) ? p : smallp;
}

template <int NDIR, bool MHD>
__device__ __forceinline__ double pthermal_raw(const double* u,
                                               const PhysConst& k) {
  const Rcp64 ir = rcp64(u[0]);
  if (MHD) return pthermal_mhd_raw<NDIR>(u, ir, k);
  return pthermal_hd_raw<NDIR>(u, ir, k);
}

// getcmax, src/vacphys0.t.mhd:79-116 (fast speed) / src/vacphys0.t.hd:72-100
template <int NDIR, bool MHD>
__device__ __forceinline__ double cmax_fn(const double* u, int idim,
                                          const PhysConst& k, double smallp) {
  typedef Lay<NDIR, MHD> L;
  const Rcp64 ir = rcp64(u[0]);
  if (MHD) {
    double p = clip_p(pthermal_mhd_raw<NDIR>(u, ir, k), smallp);
    double cs2 = div64(k.gamma * p, ir);
    double bb = u[L::B0 + 1] * u[L::B0 + 1];
#pragma unroll
    for (int c = 2; c <= NDIR; c++) bb = bb + u[L::B0 + c] * u[L::B0 + c];
    double cf2 = div64(bb, ir) + cs2;
    double bi = u[L::B0 + 1 + idim];
    // cf2*cf2 - 4*cs2*bi^2/rho
    const double q = fma(-4.0, div64(cs2 * (bi * bi), ir), cf2 * cf2);
    return sqrt(0.5 * (cf2 + sqrt(q))) + fabs(div64(u[1 + idim], ir));
  } else {
    double p = clip_p(pthermal_hd_raw<NDIR>(u, ir, k), smallp);
    double cs = sqrt(div64(k.gamma * p, ir));
    return cs + fabs(div64(u[1 + idim], ir));
  }
}

// 0.0 + x: x, with -0 made +0 (an integer select instead of an addition)
__device__ __forceinline__ double plus_zero(double x) {
  const long long b = __double_as_longlong(x);
  return b == (long long)0x8000000000000000ULL ? 0.0 : x;
}

// getflux + transport term, src/vacphys.mhd0.t:149-205 and
// src/vacphys.t.hd:49-75; the transport flux v*w is added after the
// non-transport part as in hancock/tvdmusclf (src/vactvdlf.t:67-70,220-223).
template <int NDIR, bool MHD>
__device__ __forceinline__ void flux_fn(const double* u, int idim,
                                        const PhysConst& k, double smallp,
                                        double* f) {
  typedef Lay<NDIR, MHD> L;
  const Rcp64 ir = rcp64(u[0]);
  const double v = div64(u[1 + idim], ir);
  if (MHD) {
    const double pt = ptotal_mhd<NDIR>(u, ir, k);
    const double bi = u[L::B0 + 1 + idim];
    f[0] = plus_zero(v * u[0]);
#pragma unroll
    for (int c = 1; c <= NDIR; c++) {
      double bk = u[L::B0 + c];
      double fk = (c == idim + 1) ? pt - bk * bi : -bk * bi;
      f[c] = fk + v * u[c];
    }
    double bm = u[L::B0 + 1] * u[1];
#pragma unroll
    for (int c = 2; c <= NDIR; c++) bm = bm + u[L::B0 + c] * u[c];
    f[L::E] = div64(u[1 + idim] * pt - bi * bm, ir) + v * u[L::E];
#pragma unroll
    for (int c = 1; c <= NDIR; c++) {
      if (c == idim + 1)
        f[L::B0 + c] = 0.0;
      else
        f[L::B0 + c] = div64(-u[c], ir) * bi + v * u[L::B0 + c];
    }
  } else {
    const double p = clip_p(pthermal_hd_raw<NDIR>(u, ir, k), smallp);
    f[0] = plus_zero(v * u[0]);
#pragma unroll
    for (int c = 1; c <= NDIR; c++) {
      f[c] = c == idim + 1 ? p + v * u[c] : plus_zero(v * u[c]);
    }
    f[L::E] = v * p + v * u[L::E];  // m/rho*p is v*p
  }
}

// Fortran MAX/MIN of two values, written as the same selects the CPU oracle
// uses so that even the sign of a zero result agrees.
__device__ __forceinline__ double fmax2(double a, double b) {
  return a > b ? a : b;
}
__device__ __forceinline__ double fmin2(double a, double b) {
  return a < b ? a : b;
}

// dwlimiter2, src/vacgrid.t:938-996: a = dw(i+1/2), b = dw(i-1/2)
__device__ __forceinline__ double limiter_fn(int lim, double a, double b) {
  const double s = copysign(1.0, a);
  switch (lim) {
    case LIM_WOODWARD: {
      double m = fmin2(fmin2(fabs(a), s * b), s * 0.25 * (b + a));
      return 2.0 * s * fmax2(0.0, m);
    }
    case LIM_SUPERBEE: {
      double x = fmin2(2.0 * fabs(a), s * b);
      double y = fmin2(fabs(a), 2.0 * s * b);
      return s * fmax2(fmax2(0.0, x), y);
    }
    case LIM_VANLEER:
      return 2.0 * fmax2(b * a, 0.0) / (a + b + 1.0e-12);
    case LIM_ALBADA:
      return (b * (a * a + 1.0e-12) + a * (b * b + 1.0e-12)) /
             (a * a + b * b + 2.0e-12);
    default:
      return s * fmax2(0.0, fmin2(fabs(a), s * b));
  }
}

// Half the limited slope, 0.5 * limiter_fn, with the same bits.  The selects
// and sign changes of minmod and woodward run on the integer ALUs: as
// 64-bit integers, doubles of clear sign bit compare as their values do, and
// where a and b differ in sign the result is zero.  What is left for the
// FP64 pipe is woodward's (a+b)/4 or minmod's factor 1/2, of 8 to 10
// operations (comparisons run there as well).  NaN in either operand and
// slopes that overflow take limiter_fn itself (what minmod gives for a NaN a
// and a finite b is finite, and is not left to how the selects compile).
static __device__ __noinline__ double half_limiter_fn(int lim, double a, double b) {
  return 0.5 * limiter_fn(lim, a, b);
}
__device__ __forceinline__ double hlimiter_fn(int lim, double a, double b) {
  constexpr long long SIGN = (long long)0x8000000000000000ULL;
  constexpr long long INF = 0x7ff0000000000000LL;
  const long long ia = __double_as_longlong(a);
  const long long sg = ia & SIGN;            // s = sign(1, a)
  const long long xa = ia & ~SIGN;           // |a|
  const long long xb = __double_as_longlong(b) ^ sg;  // s*b
  if (lim == LIM_WOODWARD) {
    const long long it = __double_as_longlong(0.25 * (b + a));
    const long long xt = it ^ sg;            // s*0.25*(b+a)
    long long r = xa < xb ? xa : xb;
    r = r < xt ? r : xt;
    // s*b = -0 is the smaller of the first pair, and of the second unless
    // (a+b)/4 is a zero too
    if (xb < 0) r = xb != SIGN ? 0 : xt > 0 ? SIGN : xt;
    const bool plain = (it & ~SIGN) <= INF && r < 0x7fe0000000000000LL;  // 2*r stays finite
    return plain ? __longlong_as_double(r ^ sg) : half_limiter_fn(lim, a, b);
  }
  if (lim == LIM_MINMOD) {
    long long r = xa < xb ? xa : xb;
    if (xb < 0) r = xb == SIGN ? SIGN : 0;
    return xa <= INF && (xb & ~SIGN) <= INF ? 0.5 * __longlong_as_double(r ^ sg)
                                            : half_limiter_fn(lim, a, b);
  }
  return half_limiter_fn(lim, a, b);
}

// The FP64 physics policy of the sweep templates (sweep_fp64.cu,
// roe_fp64.cu): storage and arithmetic in IEEE double.
struct PH64 {
  typedef double T;
  typedef double R;
  // 0.5 * limiter
  static __device__ __forceinline__ R hlimiter(int lim, R a, R b) {
    return hlimiter_fn(lim, a, b);
  }
  template <int NDIR, bool MHD>
  static __device__ __forceinline__ void flux(const R* u, int d,
                                              const DevPhys& k, R smallp,
                                              R* f) {
    flux_fn<NDIR, MHD>(u, d, k, smallp, f);
  }
  template <int NDIR, bool MHD>
  static __device__ __forceinline__ R cmax(const R* u, int d,
                                           const DevPhys& k, R smallp) {
    return cmax_fn<NDIR, MHD>(u, d, k, smallp);
  }
  template <int NDIR, bool MHD>
  static __device__ __forceinline__ double pthermal_raw(const R* u,
                                                        const DevPhys& k) {
    return vacgpu::pthermal_raw<NDIR, MHD>(u, k);
  }
  // dx(ix,idim) (gridsetup1, src/vacgrid.t:527-530)
  static __device__ __forceinline__ R dx(const DevArrays& a, int d, int i) {
    return a.dx[d][i];
  }
  // qdt/dx(ix,idim) of addflux (src/vacgrid.t:676-677)
  static __device__ __forceinline__ R qdx(double qdt, const DevArrays& a,
                                          int d, int i) {
    return div_dx(qdt, a, d, i);
  }
  // cmaxC*two/(dx(ixC)+dx(jxC)) (src/vactvdlf.t:188-190)
  static __device__ __forceinline__ double cfl(R cm, const DevArrays& a,
                                               int d, int i) {
    return cm * 2.0 / (a.dx[d][i] + a.dx[d][i + 1]);
  }
  // cmax/dx of getdt_courant (src/vac.t:701-702)
  static __device__ __forceinline__ double cell_ratio(R cm,
                                                      const DevArrays& a,
                                                      int d, int i) {
    return cm / a.dx[d][i];
  }
  static __device__ __forceinline__ R mul_qg(double qdt, double g) {
    return qdt * g;
  }
  static __device__ __forceinline__ R qdiv(double q) { return q; }
  // several quotients by one density, and quotients by dx(ix,idim)
  typedef Rcp64 Den;
  static __device__ __forceinline__ Den den(R b) { return rcp64(b); }
  static __device__ __forceinline__ R div(R a, const Den& r) { return div64(a, r); }
  static __device__ __forceinline__ R div_dx(R q, const DevArrays& a, int d, int i) {
    const double dx = a.dx[d][i];
    if (!a.rdx[d]) return q / dx;
    const double2 r = reinterpret_cast<const double2*>(a.rdx[d])[i];
    Rcp64 den;
    den.b = dx;
    den.y = r.x;
    den.yl = r.y;
    den.ok = exponent_within(dx, 100);
    return div64(q, den);
  }
};

}  // namespace vacgpu
