// Approximate Riemann solvers for one face (FP64).
//
// Restates get_Riemann_flux_{tvdlf,hll,hllc,hlld} (src/mod_finite_volume.t:348-729)
// and the HD HLLC helpers hd_get_lCD / hd_get_wCD (src/hd/mod_hd_hllc.t:56-257)
// for a single interface, with the reference's flux_type rules
// (src/mhd/mod_mhd_phys.t:566-589): with GLM the normal B and psi fluxes are
// "special" (taken from the left flux); without GLM the normal B uses the
// diffusive tvdlf form.
#pragma once

#include "physics.cuh"

namespace amrvac {

// An FP64 product that no later addition may be fused with.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return a * b; }

template <bool MHD, int NDIM, bool GLM>
struct FluxTypes {
  static constexpr bool bn_special = MHD && NDIM > 1 && GLM;
  static constexpr bool bn_tvdlf = MHD && NDIM > 1 && !GLM;
};

// get_Riemann_flux_tvdlf (mod_finite_volume.t:348-379)
template <class T, int NW>
__device__ __forceinline__ void riemann_tvdlf(const T *wLC, const T *wRC, const T *fL,
                                              const T *fR, T cmax, T tvdlfeps,
                                              T *F) {
  const T fac = -(T(0.5) * tvdlfeps * cmax);
#pragma unroll
  for (int v = 0; v < NW; ++v) {
    T f = T(0.5) * (fL[v] + fR[v]);
    F[v] = f + fac * (wRC[v] - wLC[v]);
  }
}

// get_Riemann_flux_hll (mod_finite_volume.t:381-437)
template <class T, bool MHD, int NDIR, bool GLM, int NDIM, int D, int FAST = 0>
__device__ __forceinline__ void riemann_hll(const T *wLC, const T *wRC, const T *fL,
                                            const T *fR, T cmax, T cmin,
                                            T tvdlfeps, T *F) {
  using V = Vars<MHD, NDIR, GLM>;
  using FT = FluxTypes<MHD, NDIM, GLM>;
  const T rden = rcp_f<FAST>(cmax - cmin);  // one reciprocal for every variable
#pragma unroll
  for (int v = 0; v < V::NW; ++v) {
    if (FT::bn_tvdlf && v == V::B0 + D) {
      F[v] = -(tvdlfeps * T(0.5) * fmax(cmax, fabs(cmin))) * (wRC[v] - wLC[v]);
    } else if (cmin >= T(0.0)) {
      F[v] = fL[v];
    } else if (cmax <= T(0.0)) {
      F[v] = fR[v];
    } else {
      F[v] = (cmax * fL[v] - cmin * fR[v] + cmin * cmax * (wRC[v] - wLC[v])) * rden;
    }
  }
}

// get_Riemann_flux_hllc (mod_finite_volume.t:439-504) + hd_get_lCD / hd_get_wCD
// (mod_hd_hllc.t:56-257); HD only, no hllcd diffusion, flathllc=.false.
// The side of the contact is chosen first, then the flux and the star state
// of that side alone are formed from its conserved (wC) and primitive (wp)
// state, every expression in the reference's order.  F = fS + c (wCD - wS)
// behind the contact, fS in a supersonic state; the HLL flux (lambda_CD
// outside the bounds) is a branch of its own.
template <class T, int NDIR, int FAST = 0>
__device__ __forceinline__ void riemann_hllc_hd(const T *wLC, const T *wRC, const T *wLp, const T *wRp, T cmax, T cmin,
                                                T *F) {
  using V = Vars<false, NDIR, false>;
  constexpr int NW = V::NW, RHO = V::RHO, MN = V::M0, E = V::E;
  auto flux = [](const T *wc, const T *w, int v) -> T {  // hd_get_flux
    if (v == RHO) return w[MN] * w[RHO];
    if (v == E) return w[MN] * (wc[E] + w[E]);
    const T f = w[MN] * wc[v];
    return v == MN ? f + w[E] : f;
  };
  const bool supl = cmin >= T(0.0), supr = cmax <= T(0.0);
  const T rden = rcp_f<FAST>(cmax - cmin);  // one reciprocal for every variable
  T whll[2];
#pragma unroll
  for (int v = 0; v < 2; ++v)
    whll[v] = (cmax * wRC[v] - cmin * wLC[v] + flux(wLC, wLp, v) - flux(wRC, wRp, v)) * rden;
  const T lam = div_f<FAST>(whll[MN], whll[RHO]);
  if (!supl && !supr && (lam >= cmax || lam <= cmin)) {  // Fhll
#pragma unroll
    for (int v = 0; v < NW; ++v)
      F[v] = (cmax * flux(wLC, wLp, v) - cmin * flux(wRC, wRp, v) + cmin * cmax * (wRC[v] - wLC[v])) * rden;
    return;
  }
  const bool right = supl ? false : (supr || lam < T(0.0) || (lam == T(0.0) && -cmin >= cmax));
  T wc[NW], w[NW], f[NW];
#pragma unroll
  for (int v = 0; v < NW; ++v) wc[v] = right ? wRC[v] : wLC[v];
  w[RHO] = wc[RHO];
  w[MN] = right ? wRp[MN] : wLp[MN];
  w[E] = right ? wRp[E] : wLp[E];
#pragma unroll
  for (int v = 0; v < NW; ++v) f[v] = flux(wc, w, v);
  if (supl || supr) {
#pragma unroll
    for (int v = 0; v < NW; ++v) F[v] = f[v];
    return;
  }
  const T cs = right ? cmax : cmin;
  const T vS = div_f<FAST>(wc[MN], wc[RHO]);
  const T csmls = rcp_f<FAST>(cs - lam);
  T wCD[NW];
  wCD[RHO] = wc[RHO] * (cs - vS) * csmls;
  wCD[MN] = wCD[RHO] * lam;
#pragma unroll
  for (int c = 1; c < NDIR; ++c) wCD[MN + c] = (cs * wc[MN + c] - f[MN + c]) * csmls;
  const T pCD = wc[RHO] * (cs - vS) * (lam - vS) + f[MN] - wc[MN] * vS;
  wCD[E] = (cs * wc[E] - f[E] + lam * pCD) * csmls;
#pragma unroll
  for (int v = 0; v < NW; ++v) F[v] = f[v] + cs * (wCD[v] - wc[v]);
}

// get_Riemann_flux_hllc (mod_finite_volume.t:439-504) + mhd_get_lCD /
// mhd_get_wCD (src/mhd/mod_mhd_hllc.t:56-241), no hllcd diffusion,
// flathllc=.false.  The star state keeps the HLL magnetic field; its flux
// has zero normal-B (and psi) entries, which the flux_type rules then
// replace by the diffusive tvdlf form without GLM, and keep with GLM (the
// reference's HLLC takes no flux_special branch).
template <class T, int NDIR, bool GLM, int NDIM, int D, int FAST = 0>
__device__ __forceinline__ void riemann_hllc_mhd(const T *wLC, const T *wRC, const T *fL, const T *fR, T cmax,
                                                 T cmin, T tvdlfeps, T *F) {
  using V = Vars<true, NDIR, GLM>;
  using FT = FluxTypes<true, NDIM, GLM>;
  constexpr int NW = V::NW, MN = V::M0 + D, BNI = V::B0 + D;
  int patchf = 1;
  if (cmin >= T(0.0)) patchf = -2;
  else if (cmax <= T(0.0)) patchf = 2;
  T whll[NW], Fhll[NW], fCD[NW];
  T lambdaCD = T(0.0);
  if (patchf == 1) {
    const T rden = rcp_f<FAST>(cmax - cmin);  // one reciprocal for every variable
#pragma unroll
    for (int v = 0; v < NW; ++v) {
      Fhll[v] = (cmax * fL[v] - cmin * fR[v] + cmin * cmax * (wRC[v] - wLC[v])) * rden;
      whll[v] = (cmax * wRC[v] - cmin * wLC[v] + fL[v] - fR[v]) * rden;
    }
    lambdaCD = div_f<FAST>(whll[MN], whll[V::RHO]);
    bool cond = true;
    if (cmin < T(0.0) && lambdaCD > T(0.0) && lambdaCD < cmax) {
      patchf = -1;
    } else if (cmax > T(0.0) && lambdaCD < T(0.0) && lambdaCD > cmin) {
      patchf = 1;
    } else if (lambdaCD >= cmax || lambdaCD <= cmin) {
      lambdaCD = T(0.0);
      patchf = 3;
      cond = false;
    }
    if (cond && lambdaCD == T(0.0)) patchf = (-cmin >= cmax) ? 1 : -1;
  }
  if (patchf == 1 || patchf == -1) {
    const bool right = (patchf == 1);
    T wSub[NW], fSub[NW];  // by value: a pointer to either side would put both in local memory
#pragma unroll
    for (int v = 0; v < NW; ++v) { wSub[v] = right ? wRC[v] : wLC[v]; fSub[v] = right ? fR[v] : fL[v]; }
    const T cspeed = right ? cmax : cmin;
    const T vSub = div_f<FAST>(wSub[MN], wSub[V::RHO]);
    const T rden = rcp_f<FAST>(cspeed - lambdaCD);  // one reciprocal for the star state
    T wCD[NW];
    wCD[V::RHO] = wSub[V::RHO] * (cspeed - vSub) * rden;
#pragma unroll
    for (int c = 0; c < NDIR; ++c) wCD[V::B0 + c] = whll[V::B0 + c];
#pragma unroll
    for (int c = 0; c < NDIR; ++c) {
      if (c != D) wCD[V::M0 + c] = (cspeed * wSub[V::M0 + c] - fSub[V::M0 + c] - wCD[BNI] * wCD[V::B0 + c]) * rden;
      else wCD[V::M0 + c] = wCD[V::RHO] * lambdaCD;
    }
    // V.B of the HLL state (summed in the order the components arrive)
    T vdb = whll[V::M0] * whll[V::B0];
#pragma unroll
    for (int c = 1; c < NDIR; ++c) vdb = vdb + whll[V::M0 + c] * whll[V::B0 + c];
    vdb = div_f<FAST>(vdb, whll[V::RHO]);
    const T pCD = wSub[V::RHO] * (cspeed - vSub) * (lambdaCD - vSub) + fSub[MN] - wSub[MN] * vSub +
                  wCD[BNI] * wCD[BNI];
    wCD[V::E] = (cspeed * wSub[V::E] - fSub[V::E] + lambdaCD * pCD - vdb * wCD[BNI]) * rden;
#pragma unroll
    for (int v = 0; v < NW; ++v) {
      if (v == BNI || (GLM && v == V::PSI)) fCD[v] = T(0.0);
      else fCD[v] = fSub[v] + cspeed * (wCD[v] - wSub[v]);
    }
  }
#pragma unroll
  for (int v = 0; v < NW; ++v) {
    if (FT::bn_tvdlf && v == BNI) {
      F[v] = -(tvdlfeps * T(0.5) * fmax(cmax, fabs(cmin))) * (wRC[v] - wLC[v]);
    } else if (patchf == -2) {
      F[v] = fL[v];
    } else if (patchf == 2) {
      F[v] = fR[v];
    } else if (patchf == 3) {
      F[v] = Fhll[v];
    } else {
      F[v] = fCD[v];
    }
  }
}

// TVD-MUSCL (fs_tvdmu) for hydrodynamics: the central flux of
// get_Riemann_flux_tvdmu (src/mod_finite_volume.t:342-346) with the
// characteristic limiter tvdlimit2 (src/mod_tvd.t:38-112) folded into the
// face flux — the Roe average hd_average, the wave speeds and jumps of
// geteigenjump2 and the right eigenvectors of rtimes2
// (src/hd/mod_hd_roe.t:58-296), entropy fix 'nul', getphi's tvdmu branch
// phi = |a qdt/dx| jump.  tvdlimit2 adds 0.5 R phi to the scaled flux
// -qdt/dx F; here F - 0.5 sum R |a| jump is returned for the same scaling.
// Rotated states: the face normal is component 0, the shear waves follow in
// the tangential components' order.
template <class T, int NDIR>
__device__ __forceinline__ void riemann_tvdmu_hd(const T *wLC, const T *wRC, const T *fL, const T *fR,
                                                 const PhysParams &P, T *F) {
  using V = Vars<false, NDIR, false>;
  constexpr int NW = V::NW;
#pragma unroll
  for (int v = 0; v < NW; ++v) F[v] = T(0.5) * (fL[v] + fR[v]);
  // hd_average
  const T qL = sqrt(wLC[V::RHO]), qR = sqrt(wRC[V::RHO]);
  const T rho = qL * qR;
  const T r = qL / qR;
  T vel[NDIR];
#pragma unroll
  for (int c = 0; c < NDIR; ++c)
    vel[c] = (wLC[V::M0 + c] / wLC[V::RHO] * r + wRC[V::M0 + c] / wRC[V::RHO]) / (T(1.0) + r);
  auto pth = [&](const T *w) {  // hd_get_pthermal
    T m2 = w[V::M0] * w[V::M0];
#pragma unroll
    for (int c = 1; c < NDIR; ++c) m2 = m2 + w[V::M0 + c] * w[V::M0 + c];
    T p = T(P.gamma - 1.0) * (w[V::E] - T(0.5) * m2 / w[V::RHO]);
    if (P.fix_small_values && p < T(P.small_pressure)) p = T(P.small_pressure);
    return p;
  };
  const T pL = pth(wLC), pR = pth(wRC);
  const T hL = (pL + wLC[V::E]) / wLC[V::RHO];
  const T hR = (pR + wRC[V::E]) / wRC[V::RHO];
  const T H = (hL * r + hR) / (T(1.0) + r);
  // geteigenjump2, il = 1 part
  T v2 = vel[0] * vel[0];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) v2 = v2 + vel[c] * vel[c];
  const T kin = T(0.5) * v2;
  T c2 = T(P.gamma - 1.0) * (H - kin);
  c2 = fmax(T(P.gamma) * T(1.0e-12) / rho, c2);  // smalldouble
  const T dpperc2 = (pR - pL) / c2;
  const T cs = sqrt(c2);
  const T dvperc = (wRC[V::M0] / wRC[V::RHO] - wLC[V::M0] / wLC[V::RHO]) / cs;
  const T u = vel[0];
  // sound waves (right, left) and the entropy wave: R columns
  const T aR = fabs(u + cs) * (T(0.5) * (dpperc2 + rho * dvperc));
  const T aL = fabs(u - cs) * (T(0.5) * (dpperc2 - rho * dvperc));
  const T aE = fabs(u) * ((-dpperc2 + wRC[V::RHO]) - wLC[V::RHO]);
  F[V::RHO] = F[V::RHO] - (T(0.5) * aR + T(0.5) * aL + T(0.5) * aE);
  F[V::E] = F[V::E] - (T(0.5) * (aR * (H + u * cs)) + T(0.5) * (aL * (H - u * cs)) + T(0.5) * (aE * kin));
  F[V::M0] = F[V::M0] - (T(0.5) * (aR * (u + cs)) + T(0.5) * (aL * (u - cs)) + T(0.5) * (aE * u));
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    // shear wave of component c: a = u, jump = rho (vR_c - vL_c)
    const T aS = fabs(u) * (rho * (wRC[V::M0 + c] / wRC[V::RHO] - wLC[V::M0 + c] / wLC[V::RHO]));
    F[V::E] = F[V::E] - T(0.5) * (aS * vel[c]);
    F[V::M0 + c] = F[V::M0 + c] - (T(0.5) * (aR * vel[c]) + T(0.5) * (aL * vel[c]) + T(0.5) * (aE * vel[c]) +
                                   T(0.5) * aS);
  }
}

// TVD-MUSCL for MHD (no GLM): the central flux with tvdlimit2's
// characteristic limiter folded in, the Roe system of src/mhd/mod_mhd_roe.t
// (average2 61-146 with arithmetic averages, geteigenjump2 160-342,
// rtimes2 355-506; divbwave on, typeentropy 'nul').  The waves are taken in
// the reference's order il = 1..nwflux: Alfven R/L, fast R/L, slow R/L, then
// (ndir 3 only: nwflux = 8) the divB and entropy waves — with ndir 2
// (nwflux = 6) the limiter loop never reaches those two.  Rotated states:
// idim = component 0, idir = 1, jdir = 2 (ndir 3) or 0 (ndir 2, where the
// reference's jdir = idir + 1 - ndir (idir / ndir) wraps to idim).
template <class T, int NDIR>
__device__ __forceinline__ void riemann_tvdmu_mhd(const T *wLC, const T *wRC, const T *fL, const T *fR,
                                                  const PhysParams &P, T *F) {
  using V = Vars<true, NDIR, false>;
  constexpr int NW = V::NW, RHO = V::RHO, E = V::E, M = V::M0, B = V::B0;
  constexpr int ID = 1, JD = NDIR == 3 ? 2 : 0;
  constexpr T smalld = T(1.0e-12);
#pragma unroll
  for (int v = 0; v < NW; ++v) F[v] = T(0.5) * (fL[v] + fR[v]);
  const T g = T(P.gamma);
  auto pth = [&](const T *w) {  // mhd_get_pthermal_origin
    T m2 = w[M] * w[M], b2 = w[B] * w[B];
#pragma unroll
    for (int c = 1; c < NDIR; ++c) { m2 = m2 + w[M + c] * w[M + c]; b2 = b2 + w[B + c] * w[B + c]; }
    T p = T(P.gamma - 1.0) * (w[E] - T(0.5) * (m2 / w[RHO] + b2));
    if (P.fix_small_values && p < T(P.small_pressure)) p = T(P.small_pressure);
    return p;
  };
  // average2
  T rho = T(0.5) * (wLC[RHO] + wRC[RHO]);
  T v[NDIR], b[NDIR], dv[NDIR], db[NDIR];
#pragma unroll
  for (int c = 0; c < NDIR; ++c) {
    v[c] = T(0.5) * (wLC[M + c] / wLC[RHO] + wRC[M + c] / wRC[RHO]);
    b[c] = T(0.5) * (wLC[B + c] + wRC[B + c]);
    dv[c] = wRC[M + c] / wRC[RHO] - wLC[M + c] / wLC[RHO];
    db[c] = wRC[B + c] - wLC[B + c];
  }
  const T pL = pth(wLC), pR = pth(wRC);
  const T pav = T(0.5) * (pL + pR);
  const T dp = pR - pL;
  const T rhodv = wRC[M] - wLC[M] - v[0] * (wRC[RHO] - wLC[RHO]);
  const T cs2 = g * pav / rho;
  T bb = b[0] * b[0];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) bb = bb + b[c] * b[c];
  T cf = bb / rho + cs2;
  T cl = T(0.5) * (cf - sqrt(cf * cf - T(4.0) * cs2 * (b[0] * b[0]) / rho));
  cf = cf - cl;
  T af = (cs2 - cl) / (cf - cl);
  af = fmin(T(1.0), fmax(af, T(0.0)));
  const T as = sqrt(T(1.0) - af);
  af = sqrt(af);
  cf = sqrt(cf);
  cl = sqrt(cl);
  rho = sqrt(rho);
  if (fabs(b[0]) < smalld) b[0] = smalld;
  if constexpr (NDIR == 2) {
    b[ID] = b[ID] >= T(0.0) ? T(1.0) : T(-1.0);
  } else {
    const T tmp = sqrt(b[1] * b[1] + b[2] * b[2]);
    if (tmp > smalld) { b[1] = b[1] / tmp; b[2] = b[2] / tmp; }
    else { b[1] = sqrt(T(0.5)); b[2] = sqrt(T(0.5)); }
  }
  const T u = v[0];
  const T sgn = copysign(T(1.0), b[0]);
  const T sqcs2 = sqrt(cs2);
  T v2 = v[0] * v[0];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) v2 = v2 + v[c] * v[c];
  const T v2a2 = T(0.5) * v2 + (T(2.0) - g) / (g - T(1.0)) * cs2;
  // Alfven waves
  const T bdvA = ((b[JD] * dv[ID] - b[ID] * dv[JD]) * T(0.5)) * (rho * rho);
  const T bdbA = ((b[JD] * db[ID] - b[ID] * db[JD]) * T(0.5)) * copysign(rho, b[0]);
  const T bvA = b[JD] * v[ID] - b[ID] * v[JD];
  // fast and slow waves
  T bdvF = b[ID] * dv[ID], bdbF = b[ID] * db[ID], bvF = b[ID] * v[ID];
  if constexpr (NDIR == 3) {
    bdvF = bdvF + b[JD] * dv[JD];
    bdbF = bdbF + b[JD] * db[JD];
    bvF = bvF + b[JD] * v[JD];
  }
  bdvF = bdvF * copysign(rho * rho, b[0]);
  bdbF = (bdbF * sqcs2) * rho;
  bvF = bvF * sgn;
  const T h = T(0.5) / cs2;
  T D[NW];
#pragma unroll
  for (int w = 0; w < NW; ++w) D[w] = T(0.0);
  // il = alfvR, alfvL, fastR, fastL, slowR, slowL (then divB, entropy for ndir 3)
#pragma unroll
  for (int il = 0; il < (NDIR == 3 ? 8 : 6); ++il) {
    T a, jump;
    switch (il) {
      case 0: a = u + fabs(b[0]) / rho; jump = bdvA - bdbA; break;
      case 1: a = u - fabs(b[0]) / rho; jump = -bdvA - bdbA; break;
      case 2: a = u + cf; jump = h * (af * (cf * rhodv + dp) + as * (-cl * bdvF + bdbF)); break;
      case 3: a = u - cf; jump = h * (af * (-cf * rhodv + dp) + as * (cl * bdvF + bdbF)); break;
      case 4: a = u + cl; jump = h * (as * (cl * rhodv + dp) + af * (cf * bdvF - bdbF)); break;
      case 5: a = u - cl; jump = h * (as * (-cl * rhodv + dp) + af * (-cf * bdvF - bdbF)); break;
      case 6: a = u; jump = db[0]; break;
      default: a = u; jump = (wRC[RHO] - wLC[RHO]) - dp / cs2; break;
    }
    const T q = fabs(a) * jump;
    const bool fast = il == 2 || il == 3, slow = il == 4 || il == 5, alf = il < 2;
    const T pm = (il == 2 || il == 4) ? T(1.0) : T(-1.0);  // R / L of fast and slow
    // rtimes2 rows
    T r_rho, r_e, r_mn, r_bn;
    if (fast) {
      r_rho = q * af;
      r_e = q * (-pm * as * cl * bvF + af * (v2a2 + cf * (cf + pm * u)));
      r_mn = (q * af) * (u + pm * cf);
    } else if (slow) {
      r_rho = q * as;
      r_e = q * (pm * af * cf * bvF + as * (v2a2 + cl * (cl + pm * u)));
      r_mn = (q * as) * (u + pm * cl);
    } else if (alf) {
      r_rho = T(0.0);
      r_e = il == 0 ? q * bvA : -q * bvA;
      r_mn = T(0.0);
    } else if (il == 6) {
      r_rho = T(0.0);
      r_e = q * b[0];
      r_mn = T(0.0);
    } else {
      r_rho = q;
      r_e = q * T(0.5) * v2;
      r_mn = q * u;
    }
    r_bn = il == 6 ? q : T(0.0);
    D[RHO] = D[RHO] + T(0.5) * r_rho;
    D[E] = D[E] + T(0.5) * r_e;
    D[M] = D[M] + T(0.5) * r_mn;
    D[B] = D[B] + T(0.5) * r_bn;
#pragma unroll
    for (int t = 1; t < NDIR; ++t) {
      T r_m, r_b;
      if (fast) {
        r_m = q * (af * v[t] - pm * as * cl * b[t] * sgn);
        r_b = ((q * as) * sqcs2) * b[t] / rho;
      } else if (slow) {
        r_m = q * (as * v[t] + pm * af * cf * b[t] * sgn);
        r_b = -((q * af) * sqcs2) * b[t] / rho;
      } else if (alf) {
        const T s = il == 0 ? T(1.0) : T(-1.0);
        r_m = t == ID ? s * q * b[JD] : -s * q * b[ID];
        r_b = t == ID ? -q * b[JD] / copysign(rho, b[0]) : q * b[ID] / copysign(rho, b[0]);
      } else if (il == 6) {
        r_m = T(0.0);
        r_b = T(0.0);
      } else {
        r_m = q * v[t];
        r_b = T(0.0);
      }
      D[M + t] = D[M + t] + T(0.5) * r_m;
      D[B + t] = D[B + t] + T(0.5) * r_b;
    }
  }
#pragma unroll
  for (int w = 0; w < NW; ++w) F[w] = F[w] - D[w];
}

// get_Riemann_flux_hlld (mod_finite_volume.t:507-729), no B0 / equilibrium
// split, from the conserved and primitive face states (rotated, after
// mhd_modify_wLR).  Both sides' one-star states enter the two-star state;
// everything behind it (physical flux, star energies, the outer Alfven
// speed) is formed for the side of the contact that the face lies in alone,
// every expression in the reference's order.
template <class T, int NDIR, bool GLM, int NDIM, int FAST = 0>
__device__ __forceinline__ void riemann_hlld(const T *wLC, const T *wRC, const T *wLp, const T *wRp, T sR, T sL, T cg,
                                             T *F) {
  using V = Vars<true, NDIR, GLM>;
  using FT = FluxTypes<true, NDIM, GLM>;
  constexpr int RHO = V::RHO, E = V::E, M = V::M0, B = V::B0;
  const T Bx = div_f<FAST>(sR * wRC[B] - sL * wLC[B], sR - sL);
  T bR2 = wRC[B] * wRC[B], bL2 = wLC[B] * wLC[B];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    bR2 = bR2 + wRC[B + c] * wRC[B + c];
    bL2 = bL2 + wLC[B + c] * wLC[B + c];
  }
  const T ptR = wRp[E] + T(0.5) * bR2;
  const T ptL = wLp[E] + T(0.5) * bL2;
  const T vR = wRp[M], vL = wLp[M];
  const T suR = (sR - vR) * wRC[RHO];
  const T suL = (sL - vL) * wLC[RHO];
  const T sm = div_f<FAST>(suR * vR - suL * vL - ptR + ptL, suR - suL);
  // one reciprocal of s - s_M per side serves the star density and energy
  const T isR = rcp_f<FAST>(sR - sm), isL = rcp_f<FAST>(sL - sm);
  const T rR = suR * isR, rL = suL * isL;
  T r1R = suR * (sR - sm) - Bx * Bx;
  if (r1R != T(0.0)) r1R = rcp_f<FAST>(r1R);
  T r1L = suL * (sL - sm) - Bx * Bx;
  if (r1L != T(0.0)) r1L = rcp_f<FAST>(r1L);
  const T pbR = (suR * (sR - vR) - Bx * Bx) * r1R;
  const T pbL = (suL * (sL - vL) - Bx * Bx) * r1L;
  const T sqR = sqrt_f<FAST>(rR), sqL = sqrt_f<FAST>(rL);
  const T tmp = rcp_f<FAST>(sqR + sqL);
  const T sg = copysign(T(1.0), Bx);
  T v1R[NDIR], v1L[NDIR], b1R[NDIR], b1L[NDIR], v2[NDIR], b2[NDIR];
  v1R[0] = v1L[0] = v2[0] = sm;
  b1R[0] = b1L[0] = b2[0] = Bx;
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    v1R[c] = wRp[M + c] - Bx * wRC[B + c] * (sm - vR) * r1R;
    v1L[c] = wLp[M + c] - Bx * wLC[B + c] * (sm - vL) * r1L;
    b1R[c] = wRC[B + c] * pbR;
    b1L[c] = wLC[B + c] * pbL;
    v2[c] = (sqL * v1L[c] + sqR * v1R[c] + (b1R[c] - b1L[c]) * sg) * tmp;
    b2[c] = (sqL * b1R[c] + sqR * b1L[c] + sqL * sqR * (v1R[c] - v1L[c]) * sg) * tmp;
  }
  const T pts = suR * (sm - vR) + ptR;
  // the side the face lies in (Miyoshi eq. 66)
  const bool supl = sL > T(0.0), left = supl || sm >= T(0.0);
  const T s = left ? sL : sR, is = left ? isL : isR, r1 = left ? rL : rR, sq = left ? sqL : sqR;
  const T pt = left ? ptL : ptR;
  const T da = div_f<FAST>(fabs(Bx), sq);
  const T s1 = left ? sm - da : sm + da;
  const bool outer = s1 >= T(0.0);
  const bool two = left ? !outer && !supl : outer;
  const bool star = left ? !supl : (outer || sR >= T(0.0));
  T wc[V::NW], w[V::NW], v1[NDIR], b1[NDIR];
#pragma unroll
  for (int v = 0; v < V::NW; ++v) {
    wc[v] = left ? wLC[v] : wRC[v];
    w[v] = left ? wLp[v] : wRp[v];
  }
#pragma unroll
  for (int c = 0; c < NDIR; ++c) {
    v1[c] = left ? v1L[c] : v1R[c];
    b1[c] = left ? b1L[c] : b1R[c];
  }
  T vb = w[M] * wc[B], v1b = v1[0] * b1[0], v2b = v2[0] * b2[0];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    vb = vb + w[M + c] * wc[B + c];
    v1b = v1b + v1[c] * b1[c];
    v2b = v2b + v2[c] * b2[c];
  }
  const T e1 = ((s - w[M]) * wc[E] - pt * w[M] + pts * sm + Bx * (vb - v1b)) * is;
  const T e2 = left ? e1 - sq * (v1b - v2b) * sg : e1 + sq * (v1b - v2b) * sg;
  T f[V::NW];
  phys_flux<T, true, NDIR, GLM, 0>(wc, w, cg, f);
  auto put = [&](T fs, T ws, T w1, T w2) -> T {
    const T t1 = fs + s * (w1 - ws);
    const T t2 = t1 + s1 * (w2 - w1);
    return two ? t2 : (star ? t1 : fs);
  };
  F[RHO] = put(f[RHO], wc[RHO], r1, r1);
  F[E] = put(f[E], wc[E], e1, e2);
#pragma unroll
  for (int c = 0; c < NDIR; ++c) {
    // star momenta rounded on their own, as the reference stores them
    F[M + c] = put(f[M + c], wc[M + c], mul_rn(v1[c], r1), mul_rn(v2[c], r1));
    F[B + c] = put(f[B + c], wc[B + c], b1[c], b2[c]);
  }
  if constexpr (GLM) F[V::PSI] = FT::bn_special ? f[V::PSI] : put(f[V::PSI], wc[V::PSI], T(0.0), T(0.0));
  if constexpr (FT::bn_special) F[B] = f[B];
}

// Where HLLD starts from the primitive states: in 3-D FP64, and in FP32 with a
// limiter that is continuous in the data.  2.5-D FP64 runs keep the reference's
// order of operations, because weakly magnetised flows there (the field loop)
// carry a last-bit difference through cada3's small slope-ratio denominators to
// 1e-8 within twenty steps; and cada3 itself jumps where tmpeta passes 1, so
// that in FP32 every rounding difference moves a few cells to the other side
// (1e-4 of the state on coarse grids).  Results there are compared with
// earlier ones more closely than that.
template <class T, int NDIM, int LIM>
constexpr bool hlld_from_primitives = sizeof(T) == 8 ? NDIM == 3 : LIM == LIM_VANLEER;

// The same solver from the primitive face states alone (rotated, after
// mhd_modify_wLR, so with GLM both sides hold the same normal field, which is
// then Bx itself): the conserved state is formed for the face's side only and
// common factors are taken out, a quarter fewer operations than riemann_hlld
// (3-D MHD 128^3 FP64 0.64 -> 0.59 ms per stage) at rounding differences.  hlld_from_primitives says where it is used.
template <class T, int NDIR, bool GLM, int NDIM, int FAST = 0>
__device__ __forceinline__ void riemann_hlld_prim(const T *wLp, const T *wRp, T sR, T sL, T cg, T inv_gamma_1, T *F) {
  using V = Vars<true, NDIR, GLM>;
  using FT = FluxTypes<true, NDIM, GLM>;
  constexpr int RHO = V::RHO, E = V::E, M = V::M0, B = V::B0;
  const T Bx = GLM ? wLp[B] : div_f<FAST>(sR * wRp[B] - sL * wLp[B], sR - sL);
  T bR2 = wRp[B] * wRp[B], bL2 = wLp[B] * wLp[B];
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    bR2 = bR2 + wRp[B + c] * wRp[B + c];
    bL2 = bL2 + wLp[B + c] * wLp[B + c];
  }
  const T ptR = wRp[E] + T(0.5) * bR2, ptL = wLp[E] + T(0.5) * bL2;
  const T dvR = sR - wRp[M], dvL = sL - wLp[M];
  const T suR = dvR * wRp[RHO], suL = dvL * wLp[RHO];
  const T sm = div_f<FAST>(suR * wRp[M] - suL * wLp[M] - ptR + ptL, suR - suL);
  const T dR = sR - sm, dL = sL - sm, Bx2 = Bx * Bx;
  // one reciprocal of s - s_M per side serves the star density and energy
  const T isR = rcp_f<FAST>(dR), isL = rcp_f<FAST>(dL);
  const T rR = suR * isR, rL = suL * isL;
  T qR = suR * dR - Bx2, qL = suL * dL - Bx2;
  // zero in an ordinary state (at rest, field along the normal, Alfven speed
  // above the sound speed): kept, as riemann_hlld does, in the fast form as
  // well.  As NaN it sent every face of a direction to the recomputation (64^3,
  // B along x, a step: cada3 FP64 612 -> 253 us, vanleer mixed 458 -> 202; with an
  // oblique field 251 -> 253 and 203 -> 202).
  qR = rcp0_f<FAST>(qR);
  qL = rcp0_f<FAST>(qL);
  const T kR = Bx * (sm - wRp[M]) * qR, kL = Bx * (sm - wLp[M]) * qL;
  const T pR = (suR * dvR - Bx2) * qR, pL = (suL * dvL - Bx2) * qL;
  const T sqR = sqrt_f<FAST>(rR), sqL = sqrt_f<FAST>(rL);
  const T tmp = rcp_f<FAST>(sqR + sqL);
  const T sg = fsign(T(1.0), Bx);
  // the side the face lies in (Miyoshi eq. 66)
  const bool supl = sL > T(0.0), left = supl || sm >= T(0.0);
  const T rho = left ? wLp[RHO] : wRp[RHO], vn = left ? wLp[M] : wRp[M], p = left ? wLp[E] : wRp[E];
  const T Bn = GLM ? Bx : (left ? wLp[B] : wRp[B]);
  const T s = left ? sL : sR, is = left ? isL : isR, dv = left ? dvL : dvR;
  const T r1 = left ? rL : rR, sq = left ? sqL : sqR, pt = left ? ptL : ptR, su = left ? suL : suR;
  const T s1 = sm + div_f<FAST>(left ? -fabs(Bx) : fabs(Bx), sq);
  const bool outer = s1 >= T(0.0);  // outside (left) / inside (right) of the Alfven wave
  const bool two = left ? !outer && !supl : outer;
  const bool star = left ? !supl : (outer || sR >= T(0.0));
  const T c1 = star ? s : T(0.0), c2 = two ? s1 : T(0.0);
  auto put = [&](T f, T d1, T d2) -> T {
    if (FAST) return f + c1 * d1 + c2 * d2;
    return two ? f + c1 * d1 + c2 * d2 : (star ? f + c1 * d1 : f);
  };
  // where w2 = w1; the product with zero carries an invalid Alfven speed into
  // every variable, as the reference's does (with FAST the others do)
  auto put1 = [&](T f, T d1) -> T { return FAST ? f + c1 * d1 : put(f, d1, T(0.0)); };
  const T m = rho * vn;
  T b2 = Bn * Bn, v2 = vn * vn, vb = vn * Bn, v1b = sm * Bx, v2b = sm * Bx;
#pragma unroll
  for (int c = 1; c < NDIR; ++c) {
    const T v1R = wRp[M + c] - wRp[B + c] * kR, v1L = wLp[M + c] - wLp[B + c] * kL;
    const T b1R = wRp[B + c] * pR, b1L = wLp[B + c] * pL;
    const T vv = (sqL * v1L + sqR * v1R + (b1R - b1L) * sg) * tmp;
    const T bb = (sqL * b1R + sqR * b1L + sqL * sqR * (v1R - v1L) * sg) * tmp;
    const T vt = left ? wLp[M + c] : wRp[M + c], bt = left ? wLp[B + c] : wRp[B + c];
    const T v1 = left ? v1L : v1R, b1 = left ? b1L : b1R;
    const T mt = rho * vt;
    F[M + c] = put(m * vt - Bn * bt, r1 * v1 - mt, r1 * (vv - v1));
    F[B + c] = put(vn * bt - Bn * vt, b1 - bt, bb - b1);
    b2 = b2 + bt * bt;
    v2 = v2 + vt * vt;
    vb = vb + vt * bt;
    v1b = v1b + v1 * b1;
    v2b = v2b + vv * bb;
  }
  const T e = p * inv_gamma_1 + T(0.5) * (v2 * rho + b2);
  const T pts = su * (sm - vn) + pt;
  const T e1 = (dv * e - pt * vn + pts * sm + Bx * (vb - v1b)) * is;
  const T de = sq * (v1b - v2b) * sg;  // w2(e) - w1(e) on the right, its negative on the left
  F[RHO] = put1(m, r1 - rho);
  F[M] = put1(m * vn - Bn * Bn + pt, r1 * sm - m);
  F[E] = put(vn * (e + pt) - Bn * vb, e1 - e, left ? -de : de);
  if constexpr (FT::bn_special) {
    F[B] = wLp[V::PSI];
    F[V::PSI] = (cg * cg) * Bx;
  } else {
    F[B] = put1(T(0.0), Bx - Bn);
    if constexpr (GLM) F[V::PSI] = put1((cg * cg) * Bx, -wLp[V::PSI]);
  }
}

}  // namespace amrvac
