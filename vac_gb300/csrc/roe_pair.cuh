// roe_pair.cuh - the face flux of 'tvdmu' with the eight-wave MHD Roe solver
// (tvdlimit2 and getphi's TVD-MUSCL branch, src/vactvd.t:86-243; average,
// geteigenjump and rtimes of src/vacphys.mhdroe.t) for two faces in packed
// FP32, so that the fused sweeps (sweep_pair.cuh, sweep_line2.cuh) run the
// Roe corrector as they run the TVDLF one.
//
// The same quantities as the split kernels' mixed solver (roe.cuh,
// average_mhd_f32): FP32 with the cancellation-free forms of the speeds and
// weights, the thermal pressures from the double-float recovery.  The eight
// waves' products R(iw,il)*|a|*jump are summed in closed form -- the fast and
// slow pairs enter a variable through their sums and differences -- so a face
// carries eight flux values, where the split kernels store 28 per face and
// read them back twice.  |a| is not normalised by dt*2/(dx(i)+dx(j)) and
// back, which cancels without an entropy fix (typeentropy 'nul' only).
// A 128x113x120 step takes 358 us (1357 on the split kernels, whose face
// records passed through memory at 23-29 % occupancy), 192^3 1041 us (5239),
// 600^2 49 us (148), 32^2 25 us (43).  The marching kernels need 220-252
// registers with it and run two CTAs per SM: they wait on the fixed latencies
// of these dependent operations, with eight warps per SM to hide them.
#pragma once
#include "pack2.cuh"

namespace vacgpu {

// lane-wise sign(b)*1, and c ? a : b with c = x >= 0 per lane
__device__ __forceinline__ f2 vsign1(f2 b) {
  f2 r;
  r.v = (b.v & 0x8000000080000000ull) | 0x3f8000003f800000ull;
  return r;
}
__device__ __forceinline__ f2 vsel_nonneg(f2 x, f2 a, f2 b) {
  float xl, xh, al, ah, bl, bh;
  f2u(x, xl, xh);
  f2u(a, al, ah);
  f2u(b, bl, bh);
  return f2m(xl >= 0.0f ? al : bl, xh >= 0.0f ? ah : bh);
}
// x > 0 ? a : b per lane
__device__ __forceinline__ f2 vsel_pos(f2 x, f2 a, f2 b) {
  float xl, xh, al, ah, bl, bh;
  f2u(x, xl, xh);
  f2u(a, al, ah);
  f2u(b, bl, bh);
  return f2m(xl > 0.0f ? al : bl, xh > 0.0f ? ah : bh);
}

// G -= sum over the waves of R(.,il)*|a(il)|*jump(il) of the faces between
// the states L and R (unclipped pressures pL, pR, inverse densities riL,
// riR): G = 2 x the numerical flux for G = F(L) + F(R).  a1, a2 receive
// |v + cf| and |v - cf| of the CFL condition.
template <int DD, int ND, typename K>
__device__ __forceinline__ void p_roe_dissipation(const f2* L, const f2* R, f2 pL, f2 pR, f2 riL,
                                                  f2 riR, const K& k, f2 c2g, bool divbwave,
                                                  f2* G, f2& a1, f2& a2) {
  constexpr int E = ND + 1, B = ND + 2;  // e; B_c is u[B + c], c from 0
  constexpr int I = (DD + 1) % ND, J = (DD + 2) % ND;
  // average: arithmetic means, the pressures clipped
  f2 v[ND], b[ND], dB[ND];
  f2 s1, s2, s3;
  const f2 dr = R[0] - L[0];
#pragma unroll
  for (int c = 0; c < ND; c++) {
    v[c] = k.half * ffma(L[1 + c], riL, R[1 + c] * riR);
    b[c] = k.half * (L[B + c] + R[B + c]);
    dB[c] = R[B + c] - L[B + c];
    const f2 dm = R[1 + c] - L[1 + c], sb = R[B + c] + L[B + c];
    s1 = c == 0 ? v[c] * dm : ffma(v[c], dm, s1);
    s2 = c == 0 ? v[c] * v[c] : ffma(v[c], v[c], s2);
    s3 = c == 0 ? dB[c] * sb : ffma(dB[c], sb, s3);
  }
  const f2 rho = k.half * (L[0] + R[0]);
  const f2 irho = vrcp(rho);
  const f2 p = k.half * (vclamp_lo(pL, k.smallp) + vclamp_lo(pR, k.smallp));
  // dp = (g-1)(de - v.dm + v^2/2 drho - d(B^2)/2)
  const f2 vv2 = k.half * s2;
  const f2 dp = k.gm1 * ffma(k.mhalf, s3, ffma(vv2, dr, (R[E] - L[E]) - s1));
  const f2 vd = v[DD];
  const f2 rdv = ffma(vd * k.mone, dr, R[1 + DD] - L[1 + DD]);
  // speeds and weights
  const f2 as2 = k.gamma * p * irho;             // sound speed^2
  f2 bt = b[I] * b[I];
  if (ND == 3) bt = ffma(b[J], b[J], bt);
  const f2 bt2 = bt * irho, ca2 = b[DD] * b[DD] * irho;
  const f2 dd = as2 - (ca2 + bt2);
  const f2 x4 = f2s(4.0f) * as2 * bt2;
  const f2 D = vsqrt(ffma(dd, dd, x4));          // cf^2 - cs^2
  const f2 zero = f2s(0.0f), one = f2s(1.0f);
  const f2 hs = vabs(dd) + D;
  // the larger of a^2-cs^2, cf^2-a^2 as a sum, the other from their product
  const f2 big = k.half * hs;
  const f2 sml = vsel_pos(hs, x4 * k.half * vrcp(hs), zero);
  const f2 iD = vsel_pos(D, vrcp(D), zero);
  const f2 na = vsel_nonneg(dd, big, sml), ns = vsel_nonneg(dd, sml, big);
  f2 af2 = vmin(one, vmax(na * iD, zero));
  f2 aw2 = vsel_pos(D, vmin(one, vmax(ns * iD, zero)), one);
  const f2 cf2 = k.half * (as2 + ca2 + bt2 + D);
  const f2 csl2 = vsel_pos(cf2, as2 * ca2 * vrcp(cf2), zero);
  const f2 cf = vsqrt(cf2), cs = vsqrt(csl2), af = vsqrt(af2), aw = vsqrt(aw2);
  const f2 sr = vsqrt(rho), isr = vrcp(sr), asnd = vsqrt(as2);
  // transverse direction, and the sign of B_d
  f2 bI, bJ;
  if (ND == 2) {
    bI = vsel_nonneg(b[I], one, f2s(-1.0f));
    bJ = zero;
  } else {
    const f2 t = vsqrt(bt);
    const f2 tc = t - f2s(1.0e-30f);
    const f2 it = vrcp(t), r2 = f2s(0.70710678f);
    bI = vsel_pos(tc, b[I] * it, r2);
    bJ = vsel_pos(tc, b[J] * it, r2);
  }
  // |B_d| below 1e-30 counts as +1e-30 (its sign must not be 0)
  const f2 bi = vsel_nonneg(vabs(b[DD]) - f2s(1.0e-30f), b[DD], f2s(1.0e-30f));
  const f2 sgn = vsign1(bi);
  // jumps: l.dw of the fast, slow and Alfven pairs
  const f2 dvI = ffma(R[1 + I], riR, (L[1 + I] * riL) * k.mone);
  f2 bdv = bI * dvI, bdb = bI * dB[I];
  f2 dvJ = zero;
  if (ND == 3) {
    dvJ = ffma(R[1 + J], riR, (L[1 + J] * riL) * k.mone);
    bdv = ffma(bJ, dvJ, bdv);
    bdb = ffma(bJ, dB[J], bdb);
  }
  bdv = bdv * (rho * sgn);
  bdb = bdb * (asnd * sr);
  const f2 ha = k.half * vrcp(as2);
  const f2 afcf = af * cf, awcs = aw * cs;
  // q: |a| * jump of the fast pair (q0, q1) and the slow pair (q2, q3)
  const f2 f0 = ffma(af, dp, aw * bdb), f1 = ffma(afcf, rdv, (awcs * bdv) * k.mone);
  const f2 g0 = ffma(aw, dp, (af * bdb) * k.mone), g1 = ffma(awcs, rdv, afcf * bdv);
  a1 = vabs(vd + cf);
  a2 = vabs(vd - cf);
  const f2 q0 = a1 * (ha * (f0 + f1)), q1 = a2 * (ha * (f0 - f1));
  const f2 q2 = vabs(vd + cs) * (ha * (g0 + g1)), q3 = vabs(vd - cs) * (ha * (g0 - g1));
  const f2 avd = vabs(vd);
  const f2 q4 = avd * ffma(dp * k.mone, vrcp(as2), dr);
  const f2 q5 = divbwave ? avd * dB[DD] : zero;
  const f2 fs = q0 + q1, fd = q0 - q1, ss = q2 + q3, sd = q2 - q3;
  // sums over the waves
  const f2 wr = ffma(af, fs, ffma(aw, ss, q4));                 // rho
  const f2 wf = afcf * fd, ws = awcs * sd;
  const f2 wt = ffma(afcf, sd, (awcs * fd) * k.mone);           // along the transverse B
  const f2 wb = (asnd * isr) * ffma(aw, fs, (af * ss) * k.mone);
  const f2 wtS = wt * sgn;
  f2 bv = bI * v[I];
  if (ND == 3) bv = ffma(bJ, v[J], bv);
  const f2 h = ffma(c2g, as2, vv2);                             // v^2/2 + (2-g)/(g-1) a^2
  f2 we = ffma(bv, wtS, h * ffma(af, fs, aw * ss));
  we = ffma(afcf, ffma(cf, fs, vd * fd), we);
  we = ffma(awcs, ffma(cs, ss, vd * sd), we);
  we = ffma(vv2, q4, ffma(bi, q5, we));
  G[0] = G[0] - wr;
  G[1 + DD] = G[1 + DD] - ffma(vd, wr, wf + ws);
  G[B + DD] = G[B + DD] - q5;
  f2 wmI = ffma(v[I], wr, bI * wtS), wbI = bI * wb;
  if (ND == 3) {
    const f2 av = (ffma(bJ, dvI, (bI * dvJ) * k.mone)) * (k.half * rho);
    const f2 ab = (ffma(bJ, dB[I], (bI * dB[J]) * k.mone)) * (k.half * sr) * sgn;
    const f2 ca = vabs(bi) * isr;
    const f2 q6 = vabs(vd + ca) * (av - ab), q7 = vabs(vd - ca) * ((av + ab) * k.mone);
    const f2 ad = q6 - q7, at = (q6 + q7) * (sgn * isr);
    const f2 bva = ffma(bJ, v[I], (bI * v[J]) * k.mone);
    we = ffma(bva, ad, we);
    wmI = ffma(bJ, ad, wmI);
    wbI = ffma(bJ * k.mone, at, wbI);
    G[1 + J] = G[1 + J] - ffma(bI * k.mone, ad, ffma(v[J], wr, bJ * wtS));
    G[B + J] = G[B + J] - ffma(bI, at, bJ * wb);
  }
  G[1 + I] = G[1 + I] - wmI;
  G[B + I] = G[B + I] - wbI;
  G[E] = G[E] - we;
}

}  // namespace vacgpu
