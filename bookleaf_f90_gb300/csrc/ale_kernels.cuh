// ale_kernels.cu -- the Eulerian remap (adv_type 1, isotropic) on sm_103a.
//
// Four kernels per ALE step replace the reference's loops of
// inf_solver_alestep (inf_solver_alestep.f90:39-74):
//   k_ale_flux    ale_kn_getmeshvelocity + geometry_kn_getvertex +
//                 geometry_kn_getfluxvolume (flux volume of every face) and the
//                 mass flux ale_kn_fluxelvl (ale_kn_sumflux(fcdv)'s sum is read
//                 by nothing).
//   k_ale_el      ale_kn_sumflux(fcdm), ale_kn_updatebasisel, the energy flux
//                 ale_kn_fluxelvl, ale_kn_fluxbasisnd (corner mass fluxes)
//                 and both momentum passes of ale_kn_fluxndvl.
//   k_ale_nd      per node: ale_kn_calcbasisnd, massbasisnd, cutbasisnd,
//                 activend and both ale_kn_updatend passes, as CSR gathers in
//                 the reference's element-major order; writes the remapped
//                 vertices (the Eulerian mesh).
//   k_ale_update  ale_kn_updateel (energy), then ale_dr_hydroupdate
//                 (geometry, density, EoS) and the new corner masses.
#pragma once
#include <cfloat>
#include <cmath>

#include "bl_device.cuh"
#include "bl_kernels.h"

namespace bl {
namespace BL_NS {

__device__ __forceinline__ bool halted_a(const DevStep* S) {
  return *((volatile const int*)&S->halted) != 0;
}

__device__ __forceinline__ int node_at(const int4& n, int j) {
  return j == 0 ? n.x : (j == 1 ? n.y : (j == 2 ? n.z : n.w));
}
__device__ __forceinline__ double cget(const d4* a, int iel, int j) {
  return reinterpret_cast<const double*>(a + iel)[j];
}

// geometry_kn_getfluxvolume for one face (before the cut)
__device__ __forceinline__ double face_dv(double x1, double x2, double y1, double y2, double x3,
                                          double x4, double y3, double y4) {
  double a1 = (-x1 - x4) + (x3 + x2);
  double a3 = (-x1 + x4) + (x3 - x2);
  double b1 = (-y1 - y4) + (y3 + y2);
  double b3 = (-y1 + y4) + (y3 - y2);
  return quarter(a1 * b3 - a3 * b1);
}

// w7 * m with w7 = SIGN(1, w) and m >= 0, and the test w1 * w2 <= 0 of the
// limiters.  The fast build takes the sign bit instead of the product (the
// same in real arithmetic: opposite signs or a zero), the exact build
// evaluates them as written.
__device__ __forceinline__ double sign_of(double m, double w) {
#if BL_FAST_ALGEBRA
  return signF(m, w);
#else
  return signF(1.0, w) * m;
#endif
}
__device__ __forceinline__ bool prod_le0(double w1, double w2) {
#if BL_FAST_ALGEBRA
  const long long b1 = bits64(w1), b2 = bits64(w2);
  return (b1 ^ b2) < 0 || (b1 << 1) == 0 || (b2 << 1) == 0;
#else
  return geF(0.0, w1 * w2);
#endif
}

#if BL_MIXED
// Mixed build: the remap limiters' gradient in FP32.  For the differences
// A, B of the advected variable towards the two neighbours and the masses
// (or volumes) mA, mB of the two sides, w8 = (A mB^2 + B mA^2) /
// (mA mB (mA + mB)) and |grad| = min(|w8|, |A|/mA, |B|/mB), zero unless A
// and B have the same sign, with the sign of S.  The operands are brought
// into FP32's range by powers of two taken from their exponents (exact),
// and the result scaled back, all on the integer pipe (f32_of, f64_of).
__device__ __forceinline__ int exp_of(double x) {
  return (int)((bits64(x) >> 52) & 0x7ff) - 1023;
}
__device__ __forceinline__ double grad_f32(double A, double B, double mA, double mB, double S) {
  if (prod_le0(A, B)) return 0.0;
  const int ev = exp_of(maxF_nn(absF(A), absF(B)));
  const int em = exp_of(maxF_nn(mA, mB));
  const float a = f32_of(A, -ev), b = f32_of(B, -ev);
  const float ma = f32_of(mA, -em), mb = f32_of(mB, -em);
  const float w8 = (a * mb * mb + b * ma * ma) / (ma * mb * (ma + mb));
  const float g = fminf(fminf(fabsf(w8), fabsf(a) / ma), fabsf(b) / mb);
  return signF(f64_of(g, ev - em), S);
}
#endif

#if BL_FAST_ALGEBRA && !BL_MIXED
// neither infinite nor a NaN
__device__ __forceinline__ bool finiteF(double x) {
  return ((unsigned)(bits64(x) >> 32) & 0x7ff00000u) != 0x7ff00000u;
}
// the leading words of an absolute value and of a value, and whether one is
// that of a positive normal number
__device__ __forceinline__ unsigned habs(double x) {
  return (unsigned)(bits64(x) >> 32) & 0x7fffffffu;
}
__device__ __forceinline__ unsigned hword(double x) { return (unsigned)(bits64(x) >> 32); }
__device__ __forceinline__ bool normal_word(unsigned h) { return h - 0x00100000u < 0x7fe00000u; }
// -1, 0 or 1 for a * b below, near (within 2^-18) or above c * d, from the
// leading words of four positive normal numbers, on the integer pipe
__device__ __forceinline__ int order_products(unsigned ha, unsigned hb, unsigned hc, unsigned hd) {
  const unsigned lo = 0x00100000u;
  const int e = (int)(ha >> 20) + (int)(hb >> 20) - (int)(hc >> 20) - (int)(hd >> 20);
  if (e > 2 || e < -2) return e > 0 ? 1 : -1;
  const unsigned long long p =
      ((unsigned long long)((ha & 0xfffffu) | lo) * ((hb & 0xfffffu) | lo)) << (2 + e);
  const unsigned long long q =
      ((unsigned long long)((hc & 0xfffffu) | lo) * ((hd & 0xfffffu) | lo)) << 2;
  const long long diff = (long long)(p - q), near = (long long)(q >> 18);
  return diff > near ? 1 : (diff < -near ? -1 : 0);
}
#endif

// The remap limiters' gradient from the differences A, B of the advected
// variable towards the two neighbours and the masses (or volumes) mA, mB of
// the two sides: zero unless A and B have the same sign, else
// min(|w8|, |A| / mA, |B| / mB) with the sign of S, w8 = (A mB^2 + B mA^2) /
// (mA mB (mA + mB)).
// Fast build: for positive mA and mB, w8 is the mean of A / mA and B / mB
// weighted by mB and mA, which lies between them, so the minimum is the
// smaller of those two quotients, and which one that is shows in the
// products A mB and B mA: one divide, no product in the FP64 pipe, where
// the three candidates took three divides and seven operations.  (Two
// divides when the products are too near to tell.)  Masses that are not
// positive, subnormal numbers, infinities and NaN take the three candidates.
__device__ __forceinline__ double slope_of_three(double A, double B, double mA, double mB,
                                                 double S) {
  const double w8 = DIV(A * mB * mB + B * mA * mA, mA * mB * (mA + mB));
  double grad = sign_of(minF(minF(absF(w8), DIV(absF(A), mA)), DIV(absF(B), mB)), S);
  if (prod_le0(A, B)) grad = 0.0;
  return grad;
}
__device__ __forceinline__ double limited_slope(double A, double B, double mA, double mB,
                                                double S) {
#if BL_MIXED
  return grad_f32(A, B, mA, mB, S);
#else
#if BL_FAST_ALGEBRA
  if (prod_le0(A, B)) return 0.0;
  const unsigned hA = habs(A), hB = habs(B), hmA = hword(mA), hmB = hword(mB);
  if (normal_word(hA) && normal_word(hB) && normal_word(hmA) && normal_word(hmB)) {
    const int o = order_products(hA, hmB, hB, hmA);
    const double q = DIV(absF(o > 0 ? B : A), o > 0 ? mB : mA);
    return signF(o == 0 ? minF_nn(q, DIV(absF(B), mB)) : q, S);
  }
#endif
  return slope_of_three(A, B, mA, mB, S);
#endif
}

// whether neither an infinity nor a NaN is among a value and four corners'
__device__ __forceinline__ bool all_finite(double v, const d4& c) {
#if BL_FAST_ALGEBRA && !BL_MIXED
  const unsigned x = max(max(habs(v), max(habs(c.x), habs(c.y))), max(habs(c.z), habs(c.w)));
  return x < 0x7ff00000u;
#else
  return true;
#endif
}

// The limited face flux of ale_kn_fluxelvl for the pair (i1, i2=i1+2),
// returning (fcflux(i1), fcflux(i2)) (ale_kn_advectors.f90:48-78).
// Fast build: where nothing leaves through a face its flux is 0 without the
// arithmetic -- unless that would be 0 times an infinity or a NaN, which the
// neighbour has to meet (finite: rv and own_b have neither).
__device__ __forceinline__ void elvl_pair(int i1, const int* nb, const int* fc,
                                          const d4* cnbasis, const double* own_b,
                                          double r1, double r2, const double* elvar,
                                          double rv, bool finite, double& o1, double& o2) {
  const int i2 = i1 + 2;
  const int iel1 = nb[i1], iel2 = nb[i2];
  const double e1 = elvar[iel1], e2 = elvar[iel2];
#if BL_FAST_ALGEBRA && !BL_MIXED
  // nothing leaves through either face, and one side has the same value, which
  // makes the slope 0 (fluid at rest; on bit patterns alone)
  const bool z1 = (bits64(r1) << 1) == 0, z2 = (bits64(r2) << 1) == 0;
  if (z1 && z2 && finite && (bits64(e1) == bits64(rv) || bits64(e2) == bits64(rv))) {
    o1 = o2 = 0.0;
    return;
  }
#endif
  const double w1 = rv - e2, w2 = e1 - rv;
  const double r3 = own_b[i2] + own_b[(i2 + 1) & 3], r4 = own_b[i1] + own_b[i1 + 1];
  const int f1 = fc[i1], f2 = fc[i2];
  const double w5 = r3 + cget(cnbasis, iel2, f2) + cget(cnbasis, iel2, (f2 + 1) & 3);
  const double w6 = r4 + cget(cnbasis, iel1, f1) + cget(cnbasis, iel1, (f1 + 1) & 3);
  const double grad = limited_slope(w1, w2, w5, w6, w2);
#if BL_FAST_ALGEBRA && !BL_MIXED
  // flow through the pair leaves through one face; the other's flux is 0
  if ((z1 || z2) && finite && finiteF(grad)) {
    const double r = z1 ? r2 : r1;
    const double o = r * fma(z1 ? negF(grad) : grad, (z1 ? r4 : r3) - half(r), rv);
    o1 = z1 ? 0.0 : o;
    o2 = z1 ? o : 0.0;
    return;
  }
#endif
  o1 = r1 * (rv + grad * (r3 - half(r1)));
  o2 = r2 * (rv - grad * (r4 - half(r2)));
}

// ================================================================ k_ale_flux

// LOOP: k_lag_state of the same step left the swept volumes of every
// element's faces 0 and 3; a face 1 or 2 takes the one of the face across it
// when that is a face 0 or 3 of the same nodes (exactly the negative), so 12
// FP64 operations a face are done once: Noh 1024x1024 1047 -> 997 us a step (with k_lag_state's
// unread results left out), the demoted form 981 -> 931, a 97x97 blast 64 -> 60.
template <int BS, bool BATCH, bool LOOP>
__global__ void __launch_bounds__(BS) k_ale_flux(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  const int4 nd = __ldg(F.ielnd + iel);
  const int4 ee = __ldg(F.ielel + iel);
  const int fcp = __ldg(F.ielfc + iel);
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted_a(S) || !ale_on(C, S)) return;
  const double dt = S->dt;
  const double zc = C.zerocut;
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  const int nb[4] = {ee.x, ee.y, ee.z, ee.w};
  const int fc[4] = {fc_of(fcp, 0), fc_of(fcp, 1), fc_of(fcp, 2), fc_of(fcp, 3)};
  double fv[4];
#if BL_FAST_ALGEBRA
  if (LOOP) {
    fv[0] = F.fdv0[iel];
    fv[3] = F.fdv3[iel];
#pragma unroll
    for (int j = 1; j <= 2; j++) {
      if (swept_across(fcp, j)) {
        fv[j] = negF((fc[j] == 0 ? F.fdv0 : F.fdv3)[nb[j]]);
      } else {
        const int a = n[j], b = n[j + 1];
        fv[j] = swept(F.ndx[a], F.ndy[a], F.ndubar[a], F.ndvbar[a], F.ndx[b], F.ndy[b],
                      F.ndubar[b], F.ndvbar[b], dt);
      }
    }
  } else {
    double x0[4], y0[4], ub[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      x0[j] = F.ndx[n[j]];
      y0[j] = F.ndy[n[j]];
      ub[j] = F.ndubar[n[j]];
      vb[j] = F.ndvbar[n[j]];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int k = (j + 1) & 3;
      fv[j] = swept(x0[j], y0[j], ub[j], vb[j], x0[k], y0[k], ub[k], vb[k], dt);
    }
  }
#else
  double x0[4], y0[4], x1[4], y1[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    x0[j] = F.ndx[n[j]];
    y0[j] = F.ndy[n[j]];
    // mesh velocity -ubar (zeul), x += dt*(-ubar)
    x1[j] = x0[j] + dt * (-F.ndubar[n[j]]);
    y1[j] = y0[j] + dt * (-F.ndvbar[n[j]]);
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int k = (j + 1) & 3;
    fv[j] = face_dv(x0[j], x0[k], y0[j], y0[k], x1[k], x1[j], y1[k], y1[j]);
  }
#endif
#pragma unroll
  for (int j = 0; j < 4; j++) fv[j] = gtF(zc, fv[j]) ? 0.0 : fv[j];
  // ale_kn_fluxelvl(cnwt, fcdv, eldensity)
  const d4 cw = F.cnwt[iel];
  const double ob[4] = {cw.x, cw.y, cw.z, cw.w};
  const double rv = F.rho[iel];
  const bool fin = all_finite(rv, cw);
  double fm[4];
  elvl_pair(0, nb, fc, F.cnwt, ob, fv[0], fv[2], F.rho, rv, fin, fm[0], fm[2]);
  elvl_pair(1, nb, fc, F.cnwt, ob, fv[1], fv[3], F.rho, rv, fin, fm[1], fm[3]);
  F.fcdm[iel] = make_d4(fm[0], fm[1], fm[2], fm[3]);
}

// ================================================================ k_ale_el

template <int BS, bool BATCH>
__global__ void __launch_bounds__(BS) k_ale_el(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  const int4 ee = __ldg(F.ielel + iel);
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted_a(S) || !ale_on(C, S)) return;
  const int nb[4] = {ee.x, ee.y, ee.z, ee.w};
  const int fcp = __ldg(F.ielfc + iel);
  const int fc[4] = {fc_of(fcp, 0), fc_of(fcp, 1), fc_of(fcp, 2), fc_of(fcp, 3)};
  const d4 fm4 = F.fcdm[iel];
  const double fm[4] = {fm4.x, fm4.y, fm4.z, fm4.w};
  // ale_kn_sumflux(fcdm): neighbour's flux of the shared face
  const double mpr = F.mass[iel];
#if BL_FAST_ALGEBRA
  // each face's net flux once: their sum is the element's gain (and four
  // times each corner's, ale_kn_fluxbasisnd), the difference of opposite
  // ones the corner mass-flux basis
  double net[4];
#pragma unroll
  for (int f = 0; f < 4; f++)
    net[f] = nb[f] == iel ? negF(fm[f]) : cget(F.fcdm, nb[f], fc[f]) - fm[f];
  const double totm = (net[0] + net[2]) + (net[1] + net[3]);
  const double cnfl = quarter(totm);
  const double c02 = quarter(net[0] - net[2]), c13 = quarter(net[1] - net[3]);
  const double cndm[4] = {c02, c13, c02, c13};
#else
  double nfm[4];
  double totm = 0.0;
#pragma unroll
  for (int i1 = 0; i1 < 2; i1++) {
    const int i2 = i1 + 2;
    double w1 = cget(F.fcdm, nb[i1], fc[i1]);
    double w2 = cget(F.fcdm, nb[i2], fc[i2]);
    nfm[i1] = w1;
    nfm[i2] = w2;
    if (nb[i1] == iel) w1 = 0.0;
    if (nb[i2] == iel) w2 = 0.0;
    totm = totm - fm[i1] - fm[i2] + w1 + w2;
  }
  // ale_kn_fluxbasisnd: corner mass-flux basis and corner mass flux
  double cndm[4], cnfl = 0.0;
#pragma unroll
  for (int i1 = 0; i1 < 2; i1++) {
    const int i2 = i1 + 2;
    double w3 = nfm[i1], w4 = nfm[i2];
    if (nb[i1] == iel) w3 = 0.0;
    if (nb[i2] == iel) w4 = 0.0;
    double w1 = w3 - fm[i1];
    double w2 = w4 - fm[i2];
    w3 = quarter(w1 - w2);
    cndm[i1] = w3;
    cndm[i2] = w3;
    w3 = quarter(w1 + w2);
    cnfl = cnfl + w3;
  }
#endif
  // ale_kn_updatebasisel: the new mass; the advected volume and its density
  // are never read (k_ale_update forms both from the remapped vertices), so
  // F.vol keeps the volume before the remap until then
  F.mpr[iel] = mpr;
  F.mass[iel] = mpr + totm;
  F.cnflux[iel] = cnfl;  // the same for the four corners
  // ale_kn_fluxelvl(cnmass, fcdm, elenergy)
  const d4 cm = F.cnmass[iel];
  const double ob[4] = {cm.x, cm.y, cm.z, cm.w};
  const double ev = F.e[iel];
  const bool fin = all_finite(ev, cm);
  double ef[4];
  elvl_pair(0, nb, fc, F.cnmass, ob, fm[0], fm[2], F.e, ev, fin, ef[0], ef[2]);
  elvl_pair(1, nb, fc, F.cnmass, ob, fm[1], fm[3], F.e, ev, fin, ef[1], ef[3]);
  F.eflux[iel] = make_d4(ef[0], ef[1], ef[2], ef[3]);
  // ale_kn_fluxndvl for u and v (ale_kn_advectors.f90:83-153): corner flux
  // pairs (ilndl, ilndr, ii) in loop order (ilfcl, icn) = (1,1),(1,2),(2,1),(2,2)
  const int4 nd = __ldg(F.ielnd + iel);
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  double cu[4], cv[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    cu[j] = F.ndu[n[j]];
    cv[j] = F.ndv[n[j]];
  }
#if BL_FAST_ALGEBRA
  double du[2][2], dv[2][2];  // the pairs' fluxes; each corner is in two pairs
#else
  double fu[4] = {0.0, 0.0, 0.0, 0.0}, fv[4] = {0.0, 0.0, 0.0, 0.0};
#endif
#pragma unroll
  for (int ilfcl = 0; ilfcl < 2; ilfcl++) {
    const int ilfcr = ilfcl + 2;
    const int iell = nb[ilfcl], ielr = nb[ilfcr];
    const int ifcl = fc[ilfcl] + 1, ifcr = fc[ilfcr] + 1;   // 1-based as in the reference
#pragma unroll
    for (int icn = 1; icn <= 2; icn++) {
      const int ilndl = ilfcl + icn - 1;                     // 0-based corners
      const int ilndr = ((ilfcr + 1) - icn + 1) % 4;
      const int ii = ilfcl + 2 * (icn - 1);
      const double cdb = cndm[ii];
      double rdu = 0.0, rdv = 0.0;
#if BL_FAST_ALGEBRA
      // Fast build: the two branches (the corner's mass flux towards the
      // left neighbour, cdb > 0, or from the right one, cdb < 0) are one
      // computation with the corners and the neighbour swapped: near is the
      // corner of the pair the limiter is centred on, far the other one,
      // and the right branch's inner and outer differences are the left
      // form's negated (exactly), so a single branch-free path serves both
      // and a warp with fluxes of both signs runs it once.
      const bool lft = gtF(cdb, 0.0);
      if (lft || gtF(0.0, cdb)) {
        const int nbe = lft ? iell : ielr;
        const int lnl = lft ? (ifcl + icn) & 3 : (ifcr + icn - 2) & 3;
        const int lnr = lft ? (ifcl - icn + 1) & 3 : (ifcr - icn - 1) & 3;
        const int nbn = node_at(__ldg(F.ielnd + nbe), lft ? lnl : lnr);
        const double rd0 = (lft ? ob[ilndl] : ob[ilndr]) - half(absF(cdb));
        const double w5 = ob[ilndl] + ob[ilndr];
        const double w6 = cget(F.cnmass, nbe, lnl) + cget(F.cnmass, nbe, lnr);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const double* cvar = q == 0 ? cu : cv;
          const double rv = lft ? cvar[ilndl] : cvar[ilndr];
          const double I = (lft ? cvar[ilndr] : cvar[ilndl]) - rv;
          const double O = rv - (q == 0 ? F.ndu : F.ndv)[nbn];
          const double grad = limited_slope(I, O, w5, w6, I);
          const double rd = cdb * (rv + grad * rd0);
          if (q == 0) rdu = rd; else rdv = rd;
        }
      }
#else
      if (gtF(cdb, 0.0)) {
        const int lnl = (ifcl + icn) % 4;
        const int lnr = (ifcl - icn + 1) % 4;
        const int4 m = __ldg(F.ielnd + iell);
        const int mm[4] = {m.x, m.y, m.z, m.w};
        double rd0 = ob[ilndl] - half(cdb);
        double w5 = ob[ilndl] + ob[ilndr];
        double w6 = cget(F.cnmass, iell, lnl) + cget(F.cnmass, iell, lnr);
        const double den = w5 * w6 * (w5 + w6);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const double* cvar = q == 0 ? cu : cv;
          const double* nvar = q == 0 ? F.ndu : F.ndv;
          double rv = cvar[ilndl];
          double w1 = rv - nvar[mm[lnl]];
          double w2 = cvar[ilndr] - rv;
          double w3 = absF(w1), w4 = absF(w2);
          double w8 = DIV(w2 * w6 * w6 + w1 * w5 * w5, den);
          double grad = sign_of(minF(minF(absF(w8), DIV(w3, w6)), DIV(w4, w5)), w2);
          if (prod_le0(w1, w2)) grad = 0.0;
          double rd = cdb * (rv + grad * rd0);
          if (q == 0) rdu = rd; else rdv = rd;
        }
      }
      if (gtF(0.0, cdb)) {
        const int lnl = (ifcr + icn - 2) % 4;
        const int lnr = (((ifcr - icn - 1) % 4) + 4) % 4;
        const int4 m = __ldg(F.ielnd + ielr);
        const int mm[4] = {m.x, m.y, m.z, m.w};
        double rd0 = ob[ilndr] + half(cdb);
        double w5 = ob[ilndl] + ob[ilndr];
        double w6 = cget(F.cnmass, ielr, lnl) + cget(F.cnmass, ielr, lnr);
        const double den = w5 * w6 * (w5 + w6);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const double* cvar = q == 0 ? cu : cv;
          const double* nvar = q == 0 ? F.ndu : F.ndv;
          double rv = cvar[ilndr];
          double w1 = rv - cvar[ilndl];
          double w2 = nvar[mm[lnr]] - rv;
          double w3 = absF(w1), w4 = absF(w2);
          double w8 = DIV(w1 * w6 * w6 + w2 * w5 * w5, den);
          double grad = -sign_of(minF(minF(absF(w8), DIV(w3, w5)), DIV(w4, w6)), w2);
          if (prod_le0(w1, w2)) grad = 0.0;
          double rd = cdb * (rv + grad * rd0);
          if (q == 0) rdu = rd; else rdv = rd;
        }
      }
#endif
#if BL_FAST_ALGEBRA
      du[ilfcl][icn - 1] = rdu;
      dv[ilfcl][icn - 1] = rdv;
#else
      fu[ilndl] = fu[ilndl] - rdu;
      fu[ilndr] = fu[ilndr] + rdu;
      fv[ilndl] = fv[ilndl] - rdv;
      fv[ilndr] = fv[ilndr] + rdv;
#endif
    }
  }
#if BL_FAST_ALGEBRA
  // pairs (left, right): (0,3), (1,2) and (1,0), (2,3); the left corner
  // loses what the right one gains
  F.cnfu[iel] = make_d4(du[1][0] - du[0][0], -(du[0][1] + du[1][0]), du[0][1] - du[1][1],
                        du[0][0] + du[1][1]);
  F.cnfv[iel] = make_d4(dv[1][0] - dv[0][0], -(dv[0][1] + dv[1][0]), dv[0][1] - dv[1][1],
                        dv[0][0] + dv[1][1]);
#else
  F.cnfu[iel] = make_d4(fu[0], fu[1], fu[2], fu[3]);
  F.cnfv[iel] = make_d4(fv[0], fv[1], fv[2], fv[3]);
#endif
}

// ================================================================ k_ale_nd

template <int BS, bool BATCH>
__global__ void __launch_bounds__(BS) k_ale_nd(DevFields F, DevCfg C) {
  const int ind = blockIdx.x * BS + threadIdx.x;
  if (ind >= F.nnd) return;
  const int b = __ldg(F.ne_off + ind), e = __ldg(F.ne_off + ind + 1);
  const DevStep* S = nd_step<BATCH>(F, ind);
  if (halted_a(S) || !ale_on(C, S)) return;
  const double dt = S->dt;
  // calcbasisnd, massbasisnd and the momentum sums in element-major
  // (ielsort2) order, each in its own sum: m1 adds the corners' mass fluxes
  // to the finished m0, so those are kept (a node of more than kKept
  // corners reads the rest again).  The quarter volumes are summed as
  // volumes, a quarter of the sum being the same bits.
  constexpr int kKept = 4;
  double v0 = 0.0, m0 = 0.0, fu = 0.0, fv = 0.0, cf[kKept];
#pragma unroll
  for (int i = 0; i < kKept; i++) {
    if (b + i < e) {
      const int c = __ldg(F.ne_ent + b + i);
      const int iel = c >> 2, j = c & 3;
      v0 = v0 + F.vol[iel];
      m0 = m0 + cget(F.cnmass, iel, j);
      cf[i] = F.cnflux[iel];
      fu = fu + cget(F.cnfu, iel, j);
      fv = fv + cget(F.cnfv, iel, j);
    }
  }
  for (int k = b + kKept; k < e; k++) {
    const int c = __ldg(F.ne_ent + k);
    const int iel = c >> 2, j = c & 3;
    v0 = v0 + F.vol[iel];
    m0 = m0 + cget(F.cnmass, iel, j);
    fu = fu + cget(F.cnfu, iel, j);
    fv = fv + cget(F.cnfv, iel, j);
  }
  v0 = quarter(v0);
  double m1 = m0;
#pragma unroll
  for (int i = 0; i < kKept; i++)
    if (b + i < e) m1 = m1 + cf[i];
  for (int k = b + kKept; k < e; k++) m1 = m1 + F.cnflux[__ldg(F.ne_ent + k) >> 2];
  const double cutm = C.dencut * v0;
  const int t = __ldg(F.indtype + ind);
  // ale_kn_activend(-1) / (-2) with indstatus = 2 (zeul)
  const bool au = (t != -1) && (t != -3);
  const bool av = (t != -2) && (t != -3);
  double u = F.ndu[ind], v = F.ndv[ind];
  if (au && gtF(m1, cutm)) u = DIV(u * m0 + fu, m1);
  if (av && gtF(m1, cutm)) v = DIV(v * m0 + fv, m1);
  F.ndu[ind] = u;
  F.ndv[ind] = v;
  // Eulerian vertex: x + dt*(-ubar)
  F.ndx[ind] = F.ndx[ind] + dt * (-F.ndubar[ind]);
  F.ndy[ind] = F.ndy[ind] + dt * (-F.ndvbar[ind]);
}

// ================================================================ k_ale_update

template <int BS, bool BATCH>
__global__ void __launch_bounds__(BS) k_ale_update(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  const int4 ee = __ldg(F.ielel + iel);
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted_a(S) || !ale_on(C, S)) return;
  const int nb[4] = {ee.x, ee.y, ee.z, ee.w};
  const int fcp = __ldg(F.ielfc + iel);
  const int fc[4] = {fc_of(fcp, 0), fc_of(fcp, 1), fc_of(fcp, 2), fc_of(fcp, 3)};
  // ale_kn_updateel: sumflux(flux) then the mass-weighted energy
  const d4 f4 = F.eflux[iel];
  const double ef[4] = {f4.x, f4.y, f4.z, f4.w};
#if BL_FAST_ALGEBRA
  double net[4];
#pragma unroll
  for (int f = 0; f < 4; f++)
    net[f] = nb[f] == iel ? negF(ef[f]) : cget(F.eflux, nb[f], fc[f]) - ef[f];
  const double elf = (net[0] + net[2]) + (net[1] + net[3]);
#else
  double elf = 0.0;
#pragma unroll
  for (int i1 = 0; i1 < 2; i1++) {
    const int i2 = i1 + 2;
    double w1 = cget(F.eflux, nb[i1], fc[i1]);
    double w2 = cget(F.eflux, nb[i2], fc[i2]);
    if (nb[i1] == iel) w1 = 0.0;
    if (nb[i2] == iel) w2 = 0.0;
    elf = elf - ef[i1] - ef[i2] + w1 + w2;
  }
#endif
  const EosTab mat = eos_tab(C, __ldg(F.ielmat + iel));
  const double m1 = F.mass[iel], mpr = F.mpr[iel];
  const double cut = F.vol[iel] * C.dencut;
  double e = F.e[iel];
  if (gtF(m1, cut)) e = DIV(e * mpr + elf, m1);
  // new corner masses (ale_kn_massbasisnd)
  const d4 cm = F.cnmass[iel];
  const double cf = F.cnflux[iel];
  F.cnmass[iel] = make_d4(cm.x + cf, cm.y + cf, cm.z + cf, cm.w + cf);
  // ale_dr_hydroupdate: geometry at the remapped vertices, density, EoS
  const int4 nd = __ldg(F.ielnd + iel);
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  double x[4], y[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    x[j] = F.ndx[n[j]];
    y[j] = F.ndy[n[j]];
  }
  Iso g = getiso(x, y);
  if (gtF(0.0, g.vol)) note_negvol(F, S, &DevStep::negvol_ale, iel + 1 - el_base<BATCH>(F, iel));
  const double rho = DIV(m1, g.vol);
  double p, cs2;
  eos_pc(C, mat, rho, e, p, cs2);
  F.a1[iel] = g.a1;
  F.a2[iel] = g.a2;
  F.a3[iel] = g.a3;
  F.b1[iel] = g.b1;
  F.b2[iel] = g.b2;
  F.b3[iel] = g.b3;
  F.cnwt[iel] = make_d4(g.w0, g.w1, g.w2, g.w3);
  F.vol[iel] = g.vol;
  F.rho[iel] = rho;
  F.e[iel] = e;
  F.p[iel] = p;
  F.cs2[iel] = cs2;
  // components are not advected; the update still refreshes their
  // geometry, density and EoS (geometry_dr_volume.f90:66-79)
  const int imx = F.elmx ? F.elmx[iel] : -1;
  if (imx >= 0) {
    const int c0 = F.imxfcp[imx], nc = F.imxncp[imx];
    for (int k = 0; k < nc; k++) {
      const int icp = c0 + k;
      const double cpv = times4(g.a1 * g.b3 - g.a3 * g.b1) * F.frvol[icp];
      const double cpr = DIV(F.cpm[icp], cpv);
      double cpp, cpc;
      eos_pc(C, __ldg(F.icpmat + icp), cpr, F.cpe[icp], cpp, cpc);
      F.cpvol[icp] = cpv;
      F.cprho[icp] = cpr;
      F.cpp[icp] = cpp;
      F.cpcs2[icp] = cpc;
    }
  }
}

static constexpr int BS_A = 128;
static constexpr int BS_AN = 64;

template <bool BATCH>
void launch_ale_t(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  const int ge = (F.nel + BS_A - 1) / BS_A;
  if (F.loop_ale) k_ale_flux<BS_A, BATCH, true><<<ge, BS_A, 0, s>>>(F, C);
  else k_ale_flux<BS_A, BATCH, false><<<ge, BS_A, 0, s>>>(F, C);
  k_ale_el<BS_A, BATCH><<<ge, BS_A, 0, s>>>(F, C);
  if constexpr (!BATCH) {
    k_ale_nd<BS_AN, false><<<(F.nnd + BS_AN - 1) / BS_AN, BS_AN, 0, s>>>(F, C);
  } else {
    // block size chosen by the batch's autotuner (128, 256 or 512)
    if (F.nd_block == 128) k_ale_nd<128, true><<<(F.nnd + 127) / 128, 128, 0, s>>>(F, C);
    else if (F.nd_block == 512) k_ale_nd<512, true><<<(F.nnd + 511) / 512, 512, 0, s>>>(F, C);
    else k_ale_nd<256, true><<<(F.nnd + 255) / 256, 256, 0, s>>>(F, C);
  }
  k_ale_update<BS_A, BATCH><<<ge, BS_A, 0, s>>>(F, C);
}
void launch_ale(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  launch_ale_t<false>(F, C, s);
}
void launch_ale_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  launch_ale_t<true>(F, C, s);
}

}  // namespace BL_NS
}  // namespace bl
