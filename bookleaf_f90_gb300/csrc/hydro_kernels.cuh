// hydro_kernels.cu -- the Lagrangian hot path on sm_103a.
//
// Five kernels per step replace the reference's sequence of loops:
//   k_edge         the three edge-viscosity loops of inf_solver_getdt
//                  (hydro_kn_edgeviscosity.f90:30-282), with utils_kn_cngather
//                  of u,v: each edge of the mesh once (fast build), each face
//                  of each element (exact build), each element (mixed build,
//                  where it is k_edgevisc).
//   k_getdt        the corner viscosities; hydro_dr_getcs2; hydro_kn_getdtcfl /
//                  getdtdiv (hydro_kn_getdt.f90:30-122) with the two
//                  argmin/argmax scans done as a block reduction plus a
//                  last-block pass that also runs time_dr_end
//                  (time_dr_advance.f90:74-132).
//   k_lag_force    inf_solver_lagstep up to the corrector force: predictor
//                  force (hydro_kn_getforce.f90), half-step vertices,
//                  geometry, density, energy, EoS, then the corrector force
//                  with hourglass and sub-zonal terms, and the mixed-cell
//                  force average (hydro_dr_getacceleration.f90:61-79).
//   k_lag_accel    hydro_kn_scatteracceleration/getacceleration/
//                  applyacceleration and utils_kn_bc per node, gathering
//                  corner contributions over a CSR in the reference's loop
//                  order; writes u^{n+1}, ubar and the final vertices.
//   k_lag_state    the corrector getstate: geometry at x^{n+1}, density,
//                  energy from e^n with the corrector forces and ubar, EoS.
//
// This file is compiled three times.  With --fmad=false (namespace exact) every
// expression keeps the reference's operand order and the results equal the CPU
// restatement bit for bit; with --fmad=true (namespace fast) the compiler may
// fuse multiply-adds and algebraic identities are used (BL_FAST_ALGEBRA);
// namespace mixed is the fast build with the edge viscosity and the limiters
// in FP32 (BL_MIXED).
#pragma once
#include <cfloat>
#include <cmath>

#include "bl_device.cuh"
#include "bl_elem.cuh"
#include "bl_fp64.cuh"
#include "bl_lreal.cuh"
#include "bl_kernels.h"
#include "bl_mma.cuh"

// The fast build may also use exact algebraic identities that can change
// only the sign of a zero (negation symmetry of opposite corners); the
// exact build evaluates every expression as written.
#ifndef BL_FAST_ALGEBRA
#define BL_FAST_ALGEBRA 0
#endif

// Every FP64 division and square root of the per-element work goes
// through the integer-pipe versions, which return the IEEE results bit for
// bit (bl_fp64.cuh); the three of the dt reduction's last block, one
// thread on the kernel's serial tail, use the hardware's (the same bits at
// a fraction of the latency).
// The divides and square roots run out of line: one body per kernel instead
// of ~60 inlined copies of ~100 instructions, which overflowed the
// instruction cache (the getdt kernels stalled on instruction fetch).
// Inlined throughout this file, a step of Sedov 512x512 takes 185.8 us against 185.8
// (fast) and 588 against 581 us (exact), k_lag_state of Noh 1024x1024 Eulerian
// 84 against 82 us; two kernels gain (DIV_IN below).
#ifndef BL_DIV_CALL
#define BL_DIV_CALL 1
#endif
#if BL_DIV_CALL
namespace bl {
static __device__ __noinline__ double ddiv_call(double a, double b) { return ddiv_rn(a, b); }
static __device__ __noinline__ double dsqrt_call(double x) { return dsqrt_rn(x); }
}  // namespace bl
#define DIV(a, b) ::bl::ddiv_call((a), (b))
#define SQRT(a) ::bl::dsqrt_call(a)
#endif
#ifndef DIV
#define DIV(a, b) ::bl::ddiv_rn((a), (b))
#endif
#ifndef SQRT
#define SQRT(a) ::bl::dsqrt_rn(a)
#endif
// Inlined divides, for k_lag_force and k_lag_accel of the fast and mixed
// builds: few enough to fit, and the independent ones (four sub-zonal
// densities; two components of an acceleration) overlap.  Called and inlined,
// a step of Sedov 301x301 in the mixed build 80.0 and 78.9 us, of 512x512 185.0
// and 183.7 (fast), 175.1 and 173.9 us (mixed), of the 300x120 polar Noh 40.0
// and 39.4 us.
#if BL_FAST_ALGEBRA
#define DIV_IN(a, b) ::bl::ddiv_rn((a), (b))
#else
#define DIV_IN(a, b) DIV(a, b)
#endif

// Resident blocks per SM that the edge and candidate kernels (of 128 threads)
// and k_lag_force (of 64) are compiled for.  All are bound by the FP64 pipe and
// wait for their integer divide chains, so warps pay until their registers run
// out: k_lag_force spills nothing at its bound, k_getdt is still faster with
// some 60 spilled values a zone at 7 blocks than without at 4.
// k_getdt at 4/5/6/7/8 blocks: Sedov 512x512 (with the edge kernel)
// 75/73/72/69/69 us; k_edge at 6/7/10/12 within 1 us of 8.  k_lag_force in
// blocks of 128, before they became 64, at 3/4/5/6: 100/90/90/91 us with
// sub-zonal and hourglass forces; five was faster by 8 % where the mesh fits one
// wave of five and not of four (280x280 to 301x301) and slower by 6 to 9 % at
// 200x200, 330x330 and 450x450.  In blocks of 64 at twice the bound (the
// registers are the same) the last wave is finer: a step of 200x200 54.7 -> 50.9
// us, of 512x512 187.6 -> 185.3 (with k_lag_state in blocks of 64 too).
#ifndef BL_GETDT_MINB
#define BL_GETDT_MINB 7
#endif
// The exact build's k_lag_force spills at any of these and gains from warps:
// 8/9/10/12 blocks 268/261/256/258 us on Sedov 512x512, 55/53/52/53 on 200x200.
#ifndef BL_FORCE_MINB
#if BL_FAST_ALGEBRA
#define BL_FORCE_MINB 8
#else
#define BL_FORCE_MINB 10
#endif
#endif
// Minimum resident blocks per SM of the two short kernels (0: the plain
// block-size bound), from sweeps of Sedov 512x512: k_lag_accel with a
// one-block bound keeps its gathers in registers (24.8 us against 26.3 us at
// the 40 registers of the plain bound); k_lag_state is best with the plain
// bound (80 registers; 1, 8, 12 and 16 blocks were slower or equal).
#ifndef BL_ACCEL_MINB
#define BL_ACCEL_MINB 1
#endif
#ifndef BL_STATE_MINB
#define BL_STATE_MINB 0
#endif
#if BL_ACCEL_MINB > 0
#define BL_ACCEL_BOUNDS(bs) __launch_bounds__(bs, BL_ACCEL_MINB)
#else
#define BL_ACCEL_BOUNDS(bs) __launch_bounds__(bs)
#endif
#if BL_STATE_MINB > 0
#define BL_STATE_BOUNDS(bs) __launch_bounds__(bs, BL_STATE_MINB)
#else
#define BL_STATE_BOUNDS(bs) __launch_bounds__(bs)
#endif

namespace bl {
namespace BL_NS {

// ------------------------------------------------------------------ EoS
// eos_kn_getpressure / eos_kn_getcs2 (eos_kn_forms.f90:28-106)
// (the material's table entries first: they hang on the material number and
// are asked for before the work whose result they meet)
struct EosTab {
  int mat, type;
  double gm1, ggm1;
};
__device__ __forceinline__ EosTab eos_tab(const DevCfg& C, int mat) {
  EosTab t;
  t.mat = mat > 0 ? mat : 0;
  t.type = __ldg(C.eos_type + t.mat);
  t.gm1 = __ldg(C.eos_gm1 + t.mat);
  t.ggm1 = __ldg(C.eos_ggm1 + t.mat);
  return t;
}
__device__ __forceinline__ void eos_pc(const DevCfg& C, const EosTab& T, double rho, double e,
                                       double& p, double& cs2) {
  const int t = T.type;
  const double* P = C.eos_param + 6 * T.mat;
  if (t == 1) {
    p = e * rho * T.gm1;
    cs2 = T.ggm1 * e;
  } else if (t == 0) {
    p = __ldg(P);
    cs2 = C.ccut;
  } else if (t == 2) {
    double t1 = DIV(rho, __ldg(P + 2));
    p = __ldg(P) * (bl_pow(t1, __ldg(P + 1)) - 1.0);
    p = maxF(p, __ldg(P + 3));
    double t2 = __ldg(P + 1) - 1.0;
    cs2 = DIV(__ldg(P) * __ldg(P + 1), __ldg(P + 2));
    cs2 = cs2 * bl_pow(t1, t2);
  } else if (t == 3) {
    double t1 = DIV(__ldg(P + 3) * __ldg(P + 5), rho);
    double t2 = DIV(__ldg(P + 4) * __ldg(P + 5), rho);
    double t3 = __ldg(P) * rho * e;
    double t4 = (1.0 - DIV(__ldg(P), t1)) * __ldg(P + 1) * bl_exp(-t1);
    double t5 = (1.0 - DIV(__ldg(P), t2)) * __ldg(P + 2) * bl_exp(-t2);
    p = t3 + t4 + t5;
    double pp = p;
    if (gt_nn(C.pcut, absF(pp))) pp = 0.0;
    double q1 = DIV(__ldg(P + 5), rho);
    double s3 = __ldg(P + 3) * q1;
    double u4 = DIV(__ldg(P), __ldg(P + 3)) + __ldg(P) * q1 - s3 * q1;
    u4 = u4 * __ldg(P + 1) * bl_exp(-s3);
    s3 = __ldg(P + 4) * q1;
    double u5 = DIV(__ldg(P), __ldg(P + 4)) + __ldg(P) * q1 - s3 * q1;
    u5 = u5 * __ldg(P + 2) * bl_exp(-s3);
    cs2 = DIV(__ldg(P) * pp, rho) + __ldg(P) * e - u4 - u5;
  } else {
    p = -1.0;
    cs2 = C.ccut;
  }
  if (gt_nn(C.pcut, absF(p))) p = 0.0;
  cs2 = maxF(cs2, C.ccut);
}

__device__ __forceinline__ void eos_pc(const DevCfg& C, int mat, double rho, double e, double& p,
                                       double& cs2) {
  eos_pc(C, eos_tab(C, mat), rho, e, p, cs2);
}

// ------------------------------------------------------------------ geometry
// geometry_kn_getiso + getvolume (geometry_kn_volume.f90:30-79)
struct Iso {
  double a1, a2, a3, b1, b2, b3, w0, w1, w2, w3, vol;
  // fast build: a1*b3 - a3*b1 and the two skew products' sum and
  // difference, T1 + T3 and T3 - T1 with T1 = a1*b2 - a2*b1 and
  // T3 = a3*b2 - a2*b3 (shared with the sub-zonal pressure force)
  double cross, ts, td;
};

#if BL_FAST_ALGEBRA
// Fast build: the same quantities with fewer roundings.  a1 and a3 share
// the diagonal differences (x2-x0) +- (x1-x3).  Expanding the reference's
// corner weights, (3b3 -+ b2)(3a1 -+ a2) - (3a3 -+ a2)(3b1 -+ b2) over 9,
// gives cross + (T3 - T1)/3, cross + (T1 + T3)/3, cross - (T3 - T1)/3,
// cross - (T1 + T3)/3 for corners 0..3 (exact in real arithmetic).
__device__ __forceinline__ void iso_volumes(Iso& g) {
  g.cross = g.a1 * g.b3 - g.a3 * g.b1;
  const double t1 = g.a1 * g.b2 - g.a2 * g.b1;
  const double t3 = g.a3 * g.b2 - g.a2 * g.b3;
  g.ts = t1 + t3;
  g.td = t3 - t1;
  const double o3 = 1.0 / 3.0;
  g.w0 = fma(g.td, o3, g.cross);
  g.w1 = fma(g.ts, o3, g.cross);
  g.w2 = fma(-g.td, o3, g.cross);
  g.w3 = fma(-g.ts, o3, g.cross);
  g.vol = times4(g.cross);
}
__device__ __forceinline__ Iso getiso(const double* x, const double* y) {
  Iso g;
  const double ux = x[2] - x[0], vx = x[1] - x[3];
  const double uy = y[2] - y[0], vy = y[1] - y[3];
  g.a1 = quarter(ux + vx);
  g.a3 = quarter(ux - vx);
  g.a2 = quarter((x[0] + x[2]) - (x[1] + x[3]));
  g.b1 = quarter(uy + vy);
  g.b3 = quarter(uy - vy);
  g.b2 = quarter((y[0] + y[2]) - (y[1] + y[3]));
  iso_volumes(g);
  return g;
}
#else
__device__ __forceinline__ Iso getiso(const double* x, const double* y) {
  Iso g;
  g.a1 = quarter(-x[0] + x[1] + x[2] - x[3]);
  g.a2 = quarter(x[0] - x[1] + x[2] - x[3]);
  g.a3 = quarter(-x[0] - x[1] + x[2] + x[3]);
  g.b1 = quarter(-y[0] + y[1] + y[2] - y[3]);
  g.b2 = quarter(y[0] - y[1] + y[2] - y[3]);
  g.b3 = quarter(-y[0] - y[1] + y[2] + y[3]);
  const double o9 = 1.0 / 9.0;
  const double A1m = 3.0 * g.a1 - g.a2, A1p = 3.0 * g.a1 + g.a2;
  const double A3m = 3.0 * g.a3 - g.a2, A3p = 3.0 * g.a3 + g.a2;
  const double B1m = 3.0 * g.b1 - g.b2, B1p = 3.0 * g.b1 + g.b2;
  const double B3m = 3.0 * g.b3 - g.b2, B3p = 3.0 * g.b3 + g.b2;
  g.w0 = o9 * (B3m * A1m - A3m * B1m);
  g.w1 = o9 * (B3p * A1m - A3p * B1m);
  g.w2 = o9 * (B3p * A1p - A3p * B1p);
  g.w3 = o9 * (B3m * A1p - A3m * B1p);
  g.vol = times4(g.a1 * g.b3 - g.a3 * g.b1);
  g.cross = g.ts = g.td = 0.0;
  return g;
}
#endif

// geometry_kn_length (geometry_kn_length.f90:99-139)
__device__ __forceinline__ double g_denom(double x1, double y1, double x2, double y2) {
  double w1 = y1 - y2, w2 = x1 - x2;
  return w1 * w1 + w2 * w2;
}
__device__ __forceinline__ double g_distpp(double x3, double y3, double x4, double y4, double x1,
                                           double y1) {
  double w1 = half(x3 + x4) - x1;
  double w2 = half(y3 + y4) - y1;
  return w1 * w1 + w2 * w2;
}
__device__ __forceinline__ double g_distpl(double x3, double y3, double x4, double y4, double x1,
                                           double y1, double x2, double y2) {
  double res = half(y1 - y2) * (x3 + x4) + half(y3 + y4) * (x2 - x1) + y2 * x1 - y1 * x2;
  return res * res;
}

// MINVAL(geometry_kn_dln(...)) (geometry_kn_length.f90:58-97)
__device__ __forceinline__ double min_dln(const double* x, const double* y, double zcut) {
  double r[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // res(k+1): denominator from corners k+2,k+3; distance of corners
    // k,k+1 midpoint... in the reference's argument order
    const int a = k, b = (k + 1) & 3, c = (k + 2) & 3, d = (k + 3) & 3;
    double w1 = g_denom(x[c], y[c], x[d], y[d]);
    if (gt_nn(zcut, w1)) r[k] = g_distpp(x[a], y[a], x[b], y[b], x[c], y[c]);
    else r[k] = DIV(g_distpl(x[a], y[a], x[b], y[b], x[c], y[c], x[d], y[d]), w1);
  }
  double m = r[0];  // all four are sums of squares or their quotients
  m = minF_nn(m, r[1]);
  m = minF_nn(m, r[2]);
  m = minF_nn(m, r[3]);
  return m;
}

#if BL_MIXED
// Mixed build: the same squared lengths from the element's iso-parametric
// coefficients.  For side k the opposite edge (corners k+2 -> k+3) is
// 2*(dx,dy) with (dx,dy) = (a1+a2, b1+b2), (a2-a3, b2-b3), (a1-a2, b1-b2),
// (a2+a3, b2+b3), and its cross product with the vector to the midpoint of
// corners k,k+1 is 4*(dx*q - dy*p) with (p,q) = (a3,b3), (a1,b1), (a3,b3),
// (a1,b1); so the reference's distpl/denom is 4 X^2 / Y with X = dx*q -
// dy*p and Y = dx^2 + dy^2 (exact in real arithmetic), and its denominator
// is 4 Y.  A degenerate opposite edge (4 Y < zcut) takes the corner form,
// for which corners(x, y) then brings the positions.
template <class T, class Q>
__device__ __forceinline__ T min_dln_iso(Q corners, T zcut, T a1, T a2, T a3, T b1, T b2, T b3) {
  const T dxs[4] = {a1 + a2, a2 - a3, a1 - a2, a2 + a3};
  const T dys[4] = {b1 + b2, b2 - b3, b1 - b2, b2 + b3};
  T r[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const T dx = dxs[k], dy = dys[k];
    const T p = (k & 1) ? a1 : a3, q = (k & 1) ? b1 : b3;
    const T Y = dx * dx + dy * dy;
    if (gt_nn(zcut, times4(Y))) {
      const int a = k, b = (k + 1) & 3, c = (k + 2) & 3;
      double x[4], y[4];
      corners(x, y);
      r[k] = (T)g_distpp(x[a], y[a], x[b], y[b], x[c], y[c]);
    } else {
      const T X = dx * q - dy * p;
      r[k] = DIV(times4(X * X), Y);
    }
  }
  T m = r[0];
  m = minF_nn(m, r[1]);
  m = minF_nn(m, r[2]);
  m = minF_nn(m, r[3]);
  return m;
}
#endif

// MINVAL(geometry_kn_dlm(...)) (geometry_kn_length.f90:30-56)
__device__ __forceinline__ double min_dlm(const double* x, const double* y) {
  double x1 = x[0] + x[1], x2 = x[2] + x[3], y1 = y[0] + y[1], y2 = y[2] + y[3];
  x1 = half(x1 - x2);
  y1 = half(y1 - y2);
  double r0 = x1 * x1 + y1 * y1;
  x1 = x[2] + x[1];
  x2 = x[0] + x[3];
  y1 = y[2] + y[1];
  y2 = y[0] + y[3];
  x1 = half(x1 - x2);
  y1 = half(y1 - y2);
  double r1 = x1 * x1 + y1 * y1;
  double m = r0;
  m = minF_nn(m, r1);
  m = minF_nn(m, r0);
  m = minF_nn(m, r1);
  return m;
}

#if !BL_FAST_ALGEBRA
// Rounding is symmetric: -a + b is a - b with the other sign, and so is a
// product with it, bit for bit -- except that a zero's sign is the
// expression's own (a - b and -a + b are both +0 where a = b).  The exact
// build negates on the integer pipe and evaluates the expression only where
// one of the sums is zero: 80 of the 480 FP64 instructions of k_lag_force
// fewer, Sedov 512x512 292 -> 268 us.
__device__ __forceinline__ bool any_zero(double a, double b, double c, double d) {
  return (bits64(a) << 1) == 0 || (bits64(b) << 1) == 0 || (bits64(c) << 1) == 0 ||
         (bits64(d) << 1) == 0;
}
#endif

// ------------------------------------------------------------------ forces
// hydro_kn_getforceP + getforceQ (hydro_kn_getforce.f90:30-71)
__device__ __forceinline__ void force_pq(double p, double a1, double a3, double b1, double b3,
                                         const d4& qx, const d4& qy, double* fx,
                                         double* fy) {
#if BL_FAST_ALGEBRA
  // opposite corners carry opposite coefficients: b3 - b1 = -(b1 - b3)
  // exactly, up to the sign of a zero.  The four sums are the ones the
  // sub-zonal pressure force uses too.
  const double db = b1 - b3, sb = b1 + b3, da = a1 - a3, sa = a1 + a3;
  fx[0] = fma(p, db, qx.x);
  fx[1] = fma(p, sb, qx.y);
  fx[2] = fma(-p, db, qx.z);
  fx[3] = fma(-p, sb, qx.w);
  fy[0] = fma(-p, da, qy.x);
  fy[1] = fma(-p, sa, qy.y);
  fy[2] = fma(p, da, qy.z);
  fy[3] = fma(p, sa, qy.w);
#else
  const double db = -b3 + b1, sb = b3 + b1, da = a3 - a1, sa = a3 + a1;
  fx[0] = p * db;
  fx[1] = p * sb;
  fy[0] = p * da;
  fy[3] = p * sa;
  fx[2] = negF(fx[0]);
  fx[3] = negF(fx[1]);
  fy[2] = negF(fy[0]);
  fy[1] = negF(fy[3]);
  if (any_zero(db, sb, da, sa)) {
    fx[2] = p * (b3 - b1);
    fx[3] = p * (-b3 - b1);
    fy[1] = p * (-a3 - a1);
    fy[2] = p * (-a3 + a1);
  }
  fx[0] = fx[0] + qx.x;
  fy[0] = fy[0] + qy.x;
  fx[1] = fx[1] + qx.y;
  fy[1] = fy[1] + qy.y;
  fx[2] = fx[2] + qx.z;
  fy[2] = fy[2] + qy.z;
  fx[3] = fx[3] + qx.w;
  fy[3] = fy[3] + qy.w;
#endif
}

#if !BL_FAST_ALGEBRA
// hydro_kn_getforceSP (hydro_kn_getforce.f90:109-188)
__device__ void force_sp(double w1, double rho, double cs2, const double* cx, const double* cy,
                         const d4& spm, double* fx, double* fy) {
  double x3 = quarter(cx[0] + cx[1] + cx[2] + cx[3]);
  double y3 = quarter(cy[0] + cy[1] + cy[2] + cy[3]);
  // edge midpoints: x2 of corner j and x4 of corner j+1 are the same sum
  // (IEEE addition commutes), so each is evaluated once
  double mx[4], my[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    mx[j] = half(cx[j] + cx[(j + 1) & 3]);
    my[j] = half(cy[j] + cy[(j + 1) & 3]);
  }
  double lfx[4][4], lfy[4][4];
#pragma unroll
  for (int j1 = 0; j1 < 4; j1++) {
    double x1 = cx[j1], y1 = cy[j1];
    double x2 = mx[j1], y2 = my[j1];
    double x4 = mx[(j1 + 3) & 3], y4 = my[(j1 + 3) & 3];
    double w3 = quarter(-x1 + x2 + x3 - x4);
    double w4 = quarter(-x1 - x2 + x3 + x4);
    double w5 = quarter(-y1 + y2 + y3 - y4);
    double w6 = quarter(-y1 - y2 + y3 + y4);
    double w2 = times4(w3 * w6 - w4 * w5);
    w2 = DIV(c4(spm, j1), w2);
    w2 = w2 - rho;
    w2 = cs2 * w2;
    const double d = w5 - w6, s = w5 + w6, dy = -w3 + w4, sy = w3 + w4;
    lfx[j1][0] = w2 * d;
    lfx[j1][1] = w2 * s;
    lfy[j1][0] = w2 * dy;
    lfy[j1][3] = w2 * sy;
    lfx[j1][2] = negF(lfx[j1][0]);
    lfx[j1][3] = negF(lfx[j1][1]);
    lfy[j1][2] = negF(lfy[j1][0]);
    lfy[j1][1] = negF(lfy[j1][3]);
    if (any_zero(d, s, dy, sy)) {
      lfx[j1][2] = w2 * (-w5 + w6);
      lfx[j1][3] = w2 * (-w5 - w6);
      lfy[j1][1] = w2 * (-w3 - w4);
      lfy[j1][2] = w2 * (w3 - w4);
    }
  }
  double w2 = half(lfx[0][3] + lfx[3][1]);
  double w3 = half(lfx[0][1] + lfx[1][3]);
  double w4 = half(lfx[1][1] + lfx[2][3]);
  double w5 = half(lfx[3][3] + lfx[2][1]);
  double w6 = quarter(lfx[0][2] + lfx[1][2] + lfx[2][2] + lfx[3][2]);
  fx[0] = fx[0] + w1 * (lfx[0][0] + w2 + w3 + w6);
  fx[1] = fx[1] + w1 * (lfx[1][0] + w4 + w3 + w6);
  fx[2] = fx[2] + w1 * (lfx[2][0] + w4 + w5 + w6);
  fx[3] = fx[3] + w1 * (lfx[3][0] + w2 + w5 + w6);
  w2 = half(lfy[0][3] + lfy[3][1]);
  w3 = half(lfy[0][1] + lfy[1][3]);
  w4 = half(lfy[1][1] + lfy[2][3]);
  w5 = half(lfy[3][3] + lfy[2][1]);
  w6 = quarter(lfy[0][2] + lfy[1][2] + lfy[2][2] + lfy[3][2]);
  fy[0] = fy[0] + w1 * (lfy[0][0] + w2 + w3 + w6);
  fy[1] = fy[1] + w1 * (lfy[1][0] + w4 + w3 + w6);
  fy[2] = fy[2] + w1 * (lfy[2][0] + w4 + w5 + w6);
  fy[3] = fy[3] + w1 * (lfy[3][0] + w2 + w5 + w6);
}
#endif

#if !BL_FAST_ALGEBRA
// hydro_kn_getforceHG (hydro_kn_getforce.f90:73-107)
__device__ __forceinline__ void force_hg(double kappa, double rho, double area, double rdt,
                                         const double* u, const double* v, double* fx,
                                         double* fy) {
  double w2 = u[0] - u[1] + u[2] - u[3];
  double w3 = v[0] - v[1] + v[2] - v[3];
  double w1 = -kappa * rho * area * rdt;
  w2 = w1 * w2;
  w3 = w1 * w3;
  fx[0] = fx[0] + w2;
  fx[1] = fx[1] - w2;
  fx[2] = fx[2] + w2;
  fx[3] = fx[3] - w2;
  fy[0] = fy[0] + w3;
  fy[1] = fy[1] - w3;
  fy[2] = fy[2] + w3;
  fy[3] = fy[3] - w3;
}
#endif

// hydro_kn_getenergy (hydro_kn_getenergy.f90:29-52): the increment w1*dt
__device__ __forceinline__ double energy_update(double e, double m, double zerocut, double dt,
                                                const double* fx, const double* fy,
                                                const double* u, const double* v) {
  double w1 = fx[0] * u[0] + fy[0] * v[0] + fx[1] * u[1] + fy[1] * v[1] + fx[2] * u[2] +
              fy[2] * v[2] + fx[3] * u[3] + fy[3] * v[3];
  w1 = -DIV(w1, maxF(m, zerocut));
  return e + w1 * dt;
}

__device__ __forceinline__ bool halted(const DevStep* S) {
  return *((volatile const int*)&S->halted) != 0;
}

// The step header of an element's or a node's mesh: the context's single
// header, or in a batch the header of the mesh it belongs to; and the first
// element of that mesh (element numbers reported to the host are local to
// their mesh).
template <bool BATCH>
__device__ __forceinline__ DevStep* el_step(const DevFields& F, int iel) {
  return BATCH ? F.steps + __ldg(F.elinst + iel) : F.step;
}
template <bool BATCH>
__device__ __forceinline__ DevStep* nd_step(const DevFields& F, int ind) {
  return BATCH ? F.steps + __ldg(F.ndinst + ind) : F.step;
}
template <bool BATCH>
__device__ __forceinline__ int el_base(const DevFields& F, int iel) {
  return BATCH ? F.inst[__ldg(F.elinst + iel)].el_begin : 0;
}

// ================================================================ k_getdt

// (value,index) pairs for the two scans.  CFL: smallest value, first index
// on ties (hydro_kn_getdt.f90:70-73).  DIV: largest value above TINY, first
// index on ties, (TINY,-1) when no element exceeds TINY (:103-116).
__device__ __forceinline__ void cfl_min(double& v, int& i, double ov, int oi) {
  const long long ko = okey(ov), kv = okey(v);
  const bool ord = !nanF(ov) && !nanF(v);
  if (ord && (ko < kv || (ko == kv && oi < i))) { v = ov; i = oi; }
}
// DIV candidates are TINY or values that exceeded it: positive, never NaN,
// so their bit patterns order as integers
__device__ __forceinline__ void div_max(double& v, int& i, double ov, int oi) {
  const long long io = bits64(ov), iv = bits64(v);
  if (io > iv || (io == iv && oi >= 0 && (i < 0 || oi < i))) { v = ov; i = oi; }
}

// How the getdt kernels read an element's connectivity and region: in the
// library's own layout (0-based rows of four, face numbers packed in one
// int).  The exact-form kernels take the layout as a parameter, so that
// bl_getdt_noalloc runs the same kernels on arrays in the reference's layout.
struct DevLayout {
  static __device__ __forceinline__ int4 nodes(const DevFields& F, int e) {
    return __ldg(F.ielnd + e);
  }
  static __device__ __forceinline__ int4 nbrs(const DevFields& F, int e) {
    return __ldg(F.ielel + e);
  }
  static __device__ __forceinline__ int faces(const DevFields& F, int e) {
    return __ldg(F.ielfc + e);
  }
  static __device__ __forceinline__ int reg(const DevFields& F, int e) {
    return __ldg(F.ielreg + e);
  }
};

// The element's squared CFL length of hydro_kn_getdtcfl (min over its
// sides of geometry_kn_dlm or _dln), or -1 for a zdtnotreg region (the
// reference's HUGE candidate); it does not depend on the viscosity.
// corners(x, y) brings the corner positions where they are needed.
// (POS: the kernels' form for coefficients that may not be the positions')
template <class L = DevLayout, bool POS = false, class Q>
__device__ __forceinline__ double getdt_cfl_len(const DevFields& F, const DevCfg& C, int iel,
                                                Q corners) {
  const int ireg = L::reg(F, iel);
  if (__ldg(C.zdtnotreg + ireg)) return -1.0;
#if BL_MIXED
  if (!POS && !__ldg(C.zmidlength + ireg))
    return from_lr(min_dln_iso<lr>(corners, lr_cut(C.zcut), to_lr(F.a1[iel]), to_lr(F.a2[iel]),
                                   to_lr(F.a3[iel]), to_lr(F.b1[iel]), to_lr(F.b2[iel]),
                                   to_lr(F.b3[iel])));
#endif
  double x[4], y[4];
  corners(x, y);
#if BL_MIXED
  if (!POS || __ldg(C.zmidlength + ireg)) return min_dlm(x, y);
  const Iso g = getiso(x, y);
  return from_lr(min_dln_iso<lr>(corners, lr_cut(C.zcut), to_lr(g.a1), to_lr(g.a2), to_lr(g.a3),
                                 to_lr(g.b1), to_lr(g.b2), to_lr(g.b3)));
#else
  return __ldg(C.zmidlength + ireg) ? min_dlm(x, y) : min_dln(x, y, C.zcut);
#endif
}

// hydro_kn_getdtdiv's candidate of the element
__device__ __forceinline__ void getdt_div(const DevFields& F, int iel, const double* u,
                                          const double* v, double& divv, int& divi) {
#if BL_MIXED
  const lr A1 = to_lr(F.a1[iel]), A3 = to_lr(F.a3[iel]), B1 = to_lr(F.b1[iel]), B3 = to_lr(F.b3[iel]);
  lr wl = to_lr(u[0]) * (-B3 + B1) + to_lr(v[0]) * (A3 - A1) + to_lr(u[1]) * (B3 + B1) +
          to_lr(v[1]) * (-A3 - A1) + to_lr(u[2]) * (B3 - B1) + to_lr(v[2]) * (-A3 + A1) +
          to_lr(u[3]) * (-B3 - B1) + to_lr(v[3]) * (A3 + A1);
  const double w1 = from_lr(DIV(absF(wl), to_lr(F.vol[iel])));
#else
  const double A1 = F.a1[iel], A3 = F.a3[iel], B1 = F.b1[iel], B3 = F.b3[iel];
  double w1 = u[0] * (-B3 + B1) + v[0] * (A3 - A1) + u[1] * (B3 + B1) + v[1] * (-A3 - A1) +
              u[2] * (B3 - B1) + v[2] * (-A3 + A1) + u[3] * (-B3 - B1) + v[3] * (A3 + A1);
  w1 = DIV(absF(w1), F.vol[iel]);
#endif
  if (gt_nn(w1, divv)) {  // divv is TINY or a larger positive value
    divv = w1;
    divi = iel;
  }
}

// hydro_dr_getcs2: elcs2 += elvisc; mixed cells: sum frmass*(cpcs2+cpvisc)
__device__ __forceinline__ double signal_speed(const DevFields& F, int iel, double cs2,
                                               double visc) {
  double cs2v = cs2 + visc;
  const int imx = F.elmx ? F.elmx[iel] : -1;
  if (imx >= 0) {
    double w1 = 0.0;
    const int c0 = F.imxfcp[imx], nc = F.imxncp[imx];
    for (int k = 0; k < nc; k++) w1 = w1 + F.frm[c0 + k] * (F.cpcs2[c0 + k] + F.cpvisc[c0 + k]);
    cs2v = w1;
  }
  F.cs2v[iel] = cs2v;
  return cs2v;
}

// the element's CFL candidate from its squared length len (getdt_cfl_len)
__device__ __forceinline__ void getdt_cfl(const DevFields& F, int iel, double len, double visc,
                                          double& cflv, int& cfli) {
  const double cs2v = signal_speed(F, iel, F.cs2[iel], visc);
#if BL_MIXED
  const double r11 = len < 0.0 ? DBL_MAX : from_lr(DIV(to_lr(len), to_lr(cs2v)));
#else
  const double r11 = len < 0.0 ? DBL_MAX : DIV(len, cs2v);
#endif
  if (cfli == 0x7fffffff) {
    cflv = r11;
    cfli = iel;
  } else {
    cfl_min(cflv, cfli, r11, iel);
  }
}

// hydro_dr_getcs2, then the element's hydro_kn_getdtcfl and getdtdiv
// candidates
template <class L = DevLayout, bool POS = false, class Q>
__device__ __forceinline__ void getdt_tail(const DevFields& F, const DevCfg& C, int iel,
                                           Q corners, const double* u, const double* v,
                                           double visc, double& cflv, int& cfli, double& divv,
                                           int& divi) {
  getdt_cfl(F, iel, getdt_cfl_len<L, POS>(F, C, iel, corners), visc, cflv, cfli);
  getdt_div(F, iel, u, v, divv, divi);
}

// A warp's smallest CFL candidate and largest divergence candidate, in every
// lane, by integer reductions: the values as order keys, high word, then low
// word among the lanes that hold it, then the first element number among
// those.  The rules are cfl_min's and div_max's; a NaN never is the smallest.
__device__ __forceinline__ void warp_cfl_min(double& v, int& i) {
  const unsigned all = 0xffffffffu;
  const unsigned long long k =
      nanF(v) ? ~0ull : (unsigned long long)okey(v) ^ 0x8000000000000000ull;
  const unsigned hi = __reduce_min_sync(all, (unsigned)(k >> 32));
  const bool h = (unsigned)(k >> 32) == hi;
  const unsigned lo = __reduce_min_sync(all, h ? (unsigned)k : all);
  const bool l = h && (unsigned)k == lo;
  const int at = __ffs(__ballot_sync(all, l)) - 1;
  i = __reduce_min_sync(all, l ? i : 0x7fffffff);
  v = from_bits64(((long long)__shfl_sync(all, (int)(bits64(v) >> 32), at) << 32) |
                  (unsigned)__shfl_sync(all, (int)bits64(v), at));
}
__device__ __forceinline__ void warp_div_max(double& v, int& i) {
  const unsigned all = 0xffffffffu;
  const unsigned long long k = (unsigned long long)bits64(v);
  const unsigned hi = __reduce_max_sync(all, (unsigned)(k >> 32));
  const bool h = (unsigned)(k >> 32) == hi;
  const unsigned lo = __reduce_max_sync(all, h ? (unsigned)k : 0u);
  const bool l = h && (unsigned)k == lo;
  const int m = __reduce_min_sync(all, l && i >= 0 ? i : 0x7fffffff);
  i = m == 0x7fffffff ? -1 : m;
  v = from_bits64((long long)(((unsigned long long)hi << 32) | lo));
}
// the same over a block, in every thread
template <int BS>
__device__ __forceinline__ void block_candidates(double& cflv, int& cfli, double& divv, int& divi,
                                                 double* s_v, int* s_i) {
  warp_cfl_min(cflv, cfli);
  warp_div_max(divv, divi);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    s_v[2 * wid] = cflv;
    s_v[2 * wid + 1] = divv;
    s_i[2 * wid] = cfli;
    s_i[2 * wid + 1] = divi;
  }
  __syncthreads();
  const int w = lane < BS / 32 ? lane : 0;
  cflv = s_v[2 * w];
  divv = s_v[2 * w + 1];
  cfli = s_i[2 * w];
  divi = s_i[2 * w + 1];
  warp_cfl_min(cflv, cfli);
  warp_div_max(divv, divi);
}

// The step header as the entry point's host reads it, written by one warp
// after its lane 0 has finished the header.
__device__ __forceinline__ void mirror_header(const DevFields& F, const DevStep* S) {
  __syncwarp();
  constexpr int N = sizeof(DevStep) / 8;
  static_assert(sizeof(DevStep) % 8 == 0 && N <= 32, "one word a lane");
  const int lane = threadIdx.x & 31;
  if (F.hstep && lane < N)
    reinterpret_cast<volatile long long*>(F.hstep)[lane] =
        reinterpret_cast<const volatile long long*>(S)[lane];
}

// The block reduction of the candidates, the last block's reduction of the
// block partials and time_dr_end (time_dr_advance.f90:74-132)
// over the k_getdt blocks [blk0, blk0 + nblk) of one mesh (all of them for
// a single mesh; a batch's mesh in a batch, whose time-step parameters then
// come from I, and whose element numbers start at el0).
// This is a serial tail that every step waits for -- on a small mesh half
// of the kernel (12,300 of 23,400 cycles at 1,000 elements) -- so it is cut
// to dependent latencies: reductions in the integer unit's warp instructions
// instead of five rounds of shuffles, one acquire-release ticket instead of
// a fence and a ticket, the step header read before the ticket, the square
// root and the divide in two warps at once, and the candidates' reciprocals
// in five lanes while the smallest is found: 7,700 cycles.
template <int BS, bool BATCH>
__device__ __forceinline__ void getdt_finish(const DevFields& F, const DevCfg& C, DevStep* S,
                                             double cflv, int cfli, double divv, int divi,
                                             int blk0, int nblk, int el0, const DevInst* I) {
  static_assert(BS >= 64 && BS / 32 <= 32, "two warps at least");
  __shared__ double s_v[2][2 * (BS / 32)], s_rdt[2];
  __shared__ int s_i[2][2 * (BS / 32)];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // the header as it is until the last block writes it
  const double dt0 = S->dt, time0 = S->time;
  const int nstep0 = S->nstep, run_mode = S->run_mode, nrec0 = S->nrecord;
  block_candidates<BS>(cflv, cfli, divv, divi, s_v[0], s_i[0]);
  if (threadIdx.x == 0) {
    reinterpret_cast<double2*>(F.red_v)[blockIdx.x] = make_double2(cflv, divv);
    reinterpret_cast<int2*>(F.red_i)[blockIdx.x] = make_int2(cfli, divi);
    unsigned int t;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(t) : "l"(&S->ticket) : "memory");
    s_last = (t == (unsigned int)(nblk - 1));
  }
  __syncthreads();
  if (!s_last) return;
  // ---- last block: reduce the partials, then time_dr_end
  cflv = HUGE_VAL;
  cfli = 0x7fffffff;
  divv = DBL_MIN;
  divi = -1;
  // Each thread takes the partials b = tid, tid + BS, ..., eight at a time:
  // their loads (L2, past the L1 that may not see other blocks' writes) are
  // all in flight before the first comparison.  (Sixteen at a time, one
  // round fewer on a 512x512 mesh, spilled in the rest of the kernel and
  // made it slower.)
  {
    constexpr int U = 8;
    const double2* rv = reinterpret_cast<const double2*>(F.red_v) + blk0;
    const int2* ri = reinterpret_cast<const int2*>(F.red_i) + blk0;
    const int nb = nblk;
    for (int b0 = threadIdx.x; b0 < nb; b0 += BS * U) {
      double2 v[U];
      int2 ix[U];
#pragma unroll
      for (int t = 0; t < U; t++) {
        const int b = b0 + t * BS;
        if (b < nb) {
          v[t] = __ldcg(rv + b);
          ix[t] = __ldcg(ri + b);
        }
      }
#pragma unroll
      for (int t = 0; t < U; t++) {
        if (b0 + t * BS < nb) {
          cfl_min(cflv, cfli, v[t].x, ix[t].x);
          div_max(divv, divi, v[t].y, ix[t].y);
        }
      }
    }
  }
  block_candidates<BS>(cflv, cfli, divv, divi, s_v[1], s_i[1]);
  // one thread's operations: the hardware's correctly rounded square root
  // and divide (the same results as the integer-pipe routines, at less
  // latency)
  if (lane == 0) {
    if (wid == 0) s_rdt[0] = C.cfl_sf * sqrt(cflv);
    else if (wid == 1) s_rdt[1] = C.div_sf / divv;
  }
  __syncthreads();
  if (wid != 0) return;
  if (lane == 0) S->ticket = 0;
  // time_dr_calc candidates then hydro's CFL and DIV (time_dr_advance.f90)
  if (cflv < 0.0) {  // hydro_kn_getdtcfl FAILURE
    if (lane == 0) {
      S->ierr = -1;
      S->iout = 2;
      S->err_code = 1;
      if (run_mode) S->halted = 1;
    }
    mirror_header(F, S);
    return;
  }
  const double rdt_cfl = s_rdt[0], rdt_div = s_rdt[1];
  const double dt_max = BATCH ? I->dt_max : C.dt_max, dt_g = BATCH ? I->dt_g : C.dt_g;
  const double dt_initial = BATCH ? I->dt_initial : C.dt_initial;
  const double dt_min = BATCH ? I->dt_min : C.dt_min, time_end = BATCH ? I->time_end : C.time_end;
  // lane k holds candidate k of the reference's order and its reciprocal
  const double g = dt_g * dt0;
  const double mine = lane == 1 ? g : lane == 2 ? dt_initial : lane == 3 ? rdt_cfl
                    : lane == 4 ? rdt_div : dt_max;
  const double inv = 1.0 / mine;
  double mind = dt_max;
  int mins = 0;
  if (gtF(mind, g)) { mind = g; mins = 1; }
  if (nstep0 == 0 && gtF(mind, dt_initial)) { mind = dt_initial; mins = 2; }
  if (gtF(mind, rdt_cfl)) { mind = rdt_cfl; mins = 3; }
  if (gtF(mind, rdt_div)) { mind = rdt_div; mins = 4; }
  const double rdt = __shfl_sync(0xffffffffu, inv, mins);
  if (lane == 0) {
    // 1-based element numbers local to the mesh (0: none)
    const int cfln = cfli >= 0 && cfli != 0x7fffffff ? cfli - el0 + 1 : 0;
    const int divn = divi >= 0 ? divi - el0 + 1 : 0;
    const int mini = mins == 3 ? cfln : (mins == 4 ? divn : -1);
    const double time = time0 + mind;
    S->cfl_rdt = rdt_cfl;
    S->cfl_idt = cfln;
    S->div_rdt = rdt_div;
    S->div_idt = divn;
    S->nstep = nstep0 + 1;
    S->dt = mind;
    S->rdt = rdt;
    S->sdt = mins;
    S->idtel = mini;
    S->time = time;
    const bool low = gtF(dt_min, mind);
    if (low) {
      S->ierr = -1;
      S->iout = 1;
      S->err_code = 2;
      if (run_mode) S->halted = 1;
    }
    if (run_mode) {
      if (geF(time, time_end)) S->stop_next = 1;
      if (F.hist && nrec0 < C.max_records) {
        StepRec& r = F.hist[nrec0];
        r.time = time;
        r.dt = mind;
        r.nstep = nstep0 + 1;
        r.idtel = mini;
        r.sdt_code = mins;
        r.ierr = low ? -1 : S->ierr;
      }
      S->nrecord = nrec0 + 1;
    }
  }
  mirror_header(F, S);
}

// Consecutive tiles of BS elements that a k_getdt block of the fast and mixed
// builds takes, for nel elements in all meshes together: about as many blocks
// as are resident at once (152 SMs of BL_GETDT_MINB), at least one tile and at
// most 8.  A block ends with a barrier and a ticket of a microsecond, which
// 8,192 blocks of one tile each pay one after another on every SM: Noh
// 1024x1024, 1, 2, 4, 8 and 16 tiles, the mixed build's k_edgevisc + k_getdt
// 203, 190, 180, 172, 196 us.  The fast build's k_getdt has FP64 work to hide
// them behind (its pair 261, 259, 258, 259, 280): the rule is the mixed
// build's, and costs the fast one nothing.  Sedov 512x512 (2,048 tiles) 1, 2
// and 4 tiles 65.3, 63.6, 67.6 us; fewer than 1.5 tiles a resident block are
// better left one each.
__host__ __device__ __forceinline__ int getdt_tiles(int nel, int bs) {
  if (!BL_FAST_ALGEBRA) return 1;
  constexpr int resident = 152 * BL_GETDT_MINB;
  const int t = (nel / bs + resident / 2) / resident;
  return t < 1 ? 1 : (t > 8 ? 8 : t);
}

#if BL_FAST_ALGEBRA
// The quantities of a face that both elements sharing it compute -- its
// lengths, unit vectors and the inverse ratio of its projections -- from
// the face's velocity (du, dv) and position (dx, dy) differences; the face
// vectors' projections on their own unit vectors are |d|^2 / max(|d|,
// zerocut) (exact in real arithmetic, never negative, so the reference's
// sign guards drop out).
// (in lr: FP64, or FP32 in the mixed build)
struct FaceQ {
  lr du, dv, lu, lx, uh, vh, xh, yh, w1;
};
__device__ __forceinline__ FaceQ face_q(lr du, lr dv, lr dx, lr dy, lr zc) {
  FaceQ f;
  f.du = du;
  f.dv = dv;
  const lr squ = du * du + dv * dv, sqx = dx * dx + dy * dy;
  f.lu = SQRT(squ);
  f.lx = SQRT(sqx);
  const lr ru = DIV((lr)1, maxF_nn(f.lu, zc)), rx = DIV((lr)1, maxF_nn(f.lx, zc));
  f.uh = du * ru;
  f.vh = dv * ru;
  f.xh = dx * rx;
  f.yh = dy * rx;
  const lr w1 = DIV(squ * ru, maxF_nn(sqx * rx, zc));
  f.w1 = DIV((lr)1, maxF_nn(w1, zc));
  return f;
}
// limiter ratio of a neighbour face with differences (ddx, ddy, ddu, ddv)
// against face f (hydro_kn_edgeviscosity.f90:117-151)
__device__ __forceinline__ lr nb_ratio(const FaceQ& f, lr ddx, lr ddy, lr ddu, lr ddv, lr zc) {
  const lr dn = ddx * f.xh + ddy * f.yh;
  const lr q = DIV(ddu * f.uh + ddv * f.vh, signF(maxF_nn(absF(dn), zc), dn));
#if BL_MIXED
  // FP32 saturates where FP64 would not: keep the ratio finite (the
  // limiter only distinguishes r below 0, in [0, 1] and above 1)
  return fmaxf(fminf(q * f.w1, 1e30f), -1e30f);
#else
  return q * f.w1;
#endif
}
#if BL_MIXED
// ================================================================ k_edgevisc

// The mixed build's edge viscosity (elvisc and the corner forces); k_getdt
// reads elvisc back.  It shares face work between neighbouring threads.
// A block of BS threads takes BS - 2 consecutive elements; thread t holds
// element blockIdx*(BS-2) + t - 1, so threads 0 and BS-1 hold the
// neighbours of the block's first and last elements (halos).  Every
// thread first publishes in shared memory the quantities of its face 0 and
// the differences of its faces 1 and 3; then each element takes
// - face 2 from the thread across it when that element is the adjacent one
//   and the face is its face 0 (the same edge run the other way: the
//   differences and unit vectors change sign, lengths and ratio do not);
// - the differences of a neighbour face of the limiter from the adjacent
//   thread when the neighbour is that element and the face is its face 1
//   or 3 (the same arithmetic on the same operands);
// and computes everything else itself, as the exact build does.  On the
// generated meshes elements are numbered along mesh lines, so the face
// across face 2 and the two limiter neighbours of side 0 are the adjacent
// elements and take the shared path.
// The FP64 build's form, one thread per edge of the mesh (k_edge), would be
// no slower here, but FP32 rounds each of an edge's two sides its own way: it
// would change results in the seventh digit, so the element form stays.
template <int BS, bool BATCH, bool POS>
__global__ void __launch_bounds__(BS, BL_GETDT_MINB) k_edgevisc(DevFields F, DevCfg C) {
  const int t = threadIdx.x;
  const int iel = (int)blockIdx.x * (BS - 2) + t - 1;
  if (!BATCH && (halted(F.step) || F.step->stop_next)) return;
  bool inmesh = iel >= 0 && iel < F.nel;
  if (BATCH && inmesh) {
    const DevStep* S = el_step<true>(F, iel);
    inmesh = !(halted(S) || S->stop_next);
  }
  const bool own = inmesh && t > 0 && t < BS - 1;
  // face 0: du dv lu lx uh vh xh yh w1, then the edge coefficient's two
  // factors that do not depend on the side the face is seen from,
  // cvisc1*sqrt((cs2 + cs2')/2) + cvisc2*|du| and rho + rho' (the same sums
  // with the operands swapped, which IEEE addition does not change)
  __shared__ lr s_f0[11][BS];
  __shared__ lr s_fd[8][BS];  // faces 1, 3: dx dy du dv each
  const lr zl = lr_cut(C.zerocut);
  int n[4] = {0, 0, 0, 0};
  double x[4], y[4], u[4], v[4];
  if (inmesh) {
    const int4 nd = __ldg(F.ielnd + iel);
    n[0] = nd.x;
    n[1] = nd.y;
    n[2] = nd.z;
    n[3] = nd.w;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      x[j] = F.ndx[n[j]];
      y[j] = F.ndy[n[j]];
      u[j] = F.ndu[n[j]];
      v[j] = F.ndv[n[j]];
    }
  }
  {
    if (inmesh) {
      const FaceQ f0 = face_q(to_lr(u[1] - u[0]), to_lr(v[1] - v[0]), to_lr(x[1] - x[0]),
                              to_lr(y[1] - y[0]), zl);
      s_f0[0][t] = f0.du;
      s_f0[1][t] = f0.dv;
      s_f0[2][t] = f0.lu;
      s_f0[3][t] = f0.lx;
      s_f0[4][t] = f0.uh;
      s_f0[5][t] = f0.vh;
      s_f0[6][t] = f0.xh;
      s_f0[7][t] = f0.yh;
      s_f0[8][t] = f0.w1;
      const int nb0 = __ldg(F.ielel + iel).x;
      s_f0[9][t] = to_lr(C.cvisc1) * SQRT(to_lr(half(F.cs2[iel] + F.cs2[nb0]))) + to_lr(C.cvisc2) * f0.lu;
      s_f0[10][t] = to_lr(F.rho[iel] + F.rho[nb0]);
      s_fd[0][t] = to_lr(x[2] - x[1]);
      s_fd[1][t] = to_lr(y[2] - y[1]);
      s_fd[2][t] = to_lr(u[2] - u[1]);
      s_fd[3][t] = to_lr(v[2] - v[1]);
      s_fd[4][t] = to_lr(x[0] - x[3]);
      s_fd[5][t] = to_lr(y[0] - y[3]);
      s_fd[6][t] = to_lr(u[0] - u[3]);
      s_fd[7][t] = to_lr(v[0] - v[3]);
    }
    __syncthreads();
  }
  if (own) {
    const double rho0 = F.rho[iel];
    // four corners of one finite velocity -- fluid at rest: every face's
    // velocity difference is 0, so its force is cut (0 <= zerocut) and its
    // viscosity 0, whatever the limiter says.  Sedov 301x301 after 60 steps
    // 78.5 -> 76.9 us a step, 512x512 174.1 -> 160.6.
    const long long ub = bits64(u[0]), vb = bits64(v[0]);
    constexpr long long kExp = 0x7FF0000000000000ll;
    const bool still = ((ub ^ bits64(u[1])) | (ub ^ bits64(u[2])) | (ub ^ bits64(u[3])) |
                        (vb ^ bits64(v[1])) | (vb ^ bits64(v[2])) | (vb ^ bits64(v[3]))) == 0 &&
                       (ub & kExp) != kExp && (vb & kExp) != kExp && zl > (lr)0 && !nanF(rho0);
    if (still) {
      F.cnviscx[iel] = make_d4(0.0, 0.0, 0.0, 0.0);
      F.cnviscy[iel] = make_d4(0.0, 0.0, 0.0, 0.0);
      F.visc[iel] = 0.0;
    } else {
      // hydro_kn_initeviscosity / limiteviscosity / geteviscosity
      // (hydro_kn_edgeviscosity.f90:30-282), face by face in the reference's
      // order 3, 1, 0, 2 (the faces of side s are (s+3)&3 and s+1)
      const int4 ee = __ldg(F.ielel + iel);
      const int nb[4] = {ee.x, ee.y, ee.z, ee.w};
      const int fcp = __ldg(F.ielfc + iel);
      const double cs2i = F.cs2[iel];
      // the vector from an edge's midpoint to the centroid is (a3,b3),
      // (-a1,-b1), (-a3,-b3), (a1,b1) for faces 0..3 (corners written as
      // s -+ a1 +- a2 -+ a3, exact in real arithmetic)
      double ca1, ca3, cb1, cb3;
      if (POS) {
        const Iso g = getiso(x, y);
        ca1 = g.a1, ca3 = g.a3, cb1 = g.b1, cb3 = g.b3;
      } else {
        ca1 = F.a1[iel], ca3 = F.a3[iel], cb1 = F.b1[iel], cb3 = F.b3[iel];
      }
      const lr ga1 = to_lr(ca1), ga3 = to_lr(ca3), gb1 = to_lr(cb1), gb3 = to_lr(cb3);
      // |c|^2 of faces 1,3 and of faces 0,2 (only the cut test uses it)
      const lr c1sq = ga1 * ga1 + gb1 * gb1, c3sq = ga3 * ga3 + gb3 * gb3;
      // max over faces of edv * |du|; the reference's max of
      // edv * 2|du| / max(rho, zerocut) is that times 2 / max(rho, zerocut)
      lr vmax = (lr)0;
      lr edx[4], edy[4];
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const int in1 = nb[s], in2 = nb[s + 2];
        const int f1 = fc_of(fcp, s), f2 = fc_of(fcp, s + 2);
        // boundary rule (hydro_kn_edgeviscosity.f90:154-183)
        lr val1 = (lr)0, val2 = (lr)0;
        if (in1 == iel)
          val1 = (__ldg(F.indtype + n[s]) < 0 && __ldg(F.indtype + n[(s + 1) & 3]) < 0 && in2 != iel)
                     ? (lr)1 : (lr)0;
        if (in2 == iel)
          val2 = (__ldg(F.indtype + n[s + 2]) < 0 && __ldg(F.indtype + n[(s + 3) & 3]) < 0 &&
                  in1 != iel) ? (lr)1 : (lr)0;
#pragma unroll
        for (int e2 = 0; e2 < 2; e2++) {
          const int is = e2 == 0 ? ((s + 3) & 3) : (s + 1);
          FaceQ f;
          int qf = -1;  // thread whose face-0 coefficient factors apply
          if (is == 0) {
            qf = t;
            f.du = s_f0[0][t];
            f.dv = s_f0[1][t];
            f.lu = s_f0[2][t];
            f.lx = s_f0[3][t];
            f.uh = s_f0[4][t];
            f.vh = s_f0[5][t];
            f.xh = s_f0[6][t];
            f.yh = s_f0[7][t];
            f.w1 = s_f0[8][t];
          } else if (is == 2) {
            const int o = nb[2] - iel;
            if ((o == 1 || o == -1) && fc_of(fcp, 2) == 0) {
              const int q = t + o;
              qf = q;
              f.du = negF(s_f0[0][q]);
              f.dv = negF(s_f0[1][q]);
              f.lu = s_f0[2][q];
              f.lx = s_f0[3][q];
              f.uh = negF(s_f0[4][q]);
              f.vh = negF(s_f0[5][q]);
              f.xh = negF(s_f0[6][q]);
              f.yh = negF(s_f0[7][q]);
              f.w1 = s_f0[8][q];
            } else {
              f = face_q(to_lr(u[3] - u[2]), to_lr(v[3] - v[2]), to_lr(x[3] - x[2]),
                         to_lr(y[3] - y[2]), zl);
            }
          } else {
            const int o = is == 1 ? 0 : 4;
            f = face_q(s_fd[o + 2][t], s_fd[o + 3][t], s_fd[o][t], s_fd[o + 1][t], zl);
          }
          // neighbour faces: edge 1 uses MOD(ielfc,4)+1 / MOD(ielfc+2,4)+1,
          // edge 2 the other pair (hydro_kn_edgeviscosity.f90:117-151)
          const int ins1 = e2 == 0 ? ((f1 + 1) & 3) : ((f1 + 3) & 3);
          const int ins2 = e2 == 0 ? ((f2 + 3) & 3) : ((f2 + 1) & 3);
          lr r1 = val1, r2 = val2;
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const int inb = k == 0 ? in1 : in2;
            const int ins = k == 0 ? ins1 : ins2;
            if (inb == iel) continue;
            lr ddx, ddy, ddu, ddv;
            const int o = inb - iel;
            if ((o == 1 || o == -1) && (ins & 1)) {
              const int q = t + o, c = ins == 1 ? 0 : 4;
              ddx = s_fd[c][q];
              ddy = s_fd[c + 1][q];
              ddu = s_fd[c + 2][q];
              ddv = s_fd[c + 3][q];
            } else {
              const int4 m = __ldg(F.ielnd + inb);
              const int mm[4] = {m.x, m.y, m.z, m.w};
              const int a = mm[ins], b = mm[(ins + 1) & 3];
              ddx = to_lr(F.ndx[b] - F.ndx[a]);
              ddy = to_lr(F.ndy[b] - F.ndy[a]);
              ddu = to_lr(F.ndu[b] - F.ndu[a]);
              ddv = to_lr(F.ndv[b] - F.ndv[a]);
            }
            const lr r = nb_ratio(f, ddx, ddy, ddu, ddv, zl);
            if (k == 0) r1 = r;
            else r2 = r;
          }
          // limiter and edge coefficient (hydro_kn_edgeviscosity.f90:185-214)
          lr cq, rs;
          if (qf >= 0) {
            cq = s_f0[9][qf];
            rs = s_f0[10][qf];
          } else {
            const int ins = nb[is];
            cq = to_lr(C.cvisc1) * SQRT(to_lr(half(cs2i + F.cs2[ins]))) + to_lr(C.cvisc2) * f.lu;
            rs = to_lr(rho0 + F.rho[ins]);
          }
          lr w2 = minF(minF(minF(half(r1 + r2), twice(r1)), twice(r2)), (lr)1);
          w2 = maxF((lr)0, w2);
          const lr edv = half((lr)1 - w2) * rs * cq;
          vmax = maxF_nn(vmax, edv * f.lu);  // never negative
          // edge force (hydro_kn_edgeviscosity.f90:219-282): the reference
          // normalises the midpoint-to-centroid vector c, orients it by the
          // sign of its product with the face vector and scales it back by
          // |c|: (exh, eyh) = -+(cy, -cx), the sign bit of w33 = cy*xh -
          // cx*yh choosing; |c| only enters the cut test
          const lr cx = is == 0 ? ga3 : (is == 1 ? negF(ga1) : (is == 2 ? negF(ga3) : ga1));
          const lr cy = is == 0 ? gb3 : (is == 1 ? negF(gb1) : (is == 2 ? negF(gb3) : gb1));
          const lr w33 = cy * f.xh - cx * f.yh;
          const lr exh = negxorsign(cy, w33);
          const lr eyh = xorsign(cx, w33);
          const lr w7sq = (is & 1) ? c1sq : c3sq;
          const lr w6b = f.du * exh + f.dv * eyh;
          const lr d = edv * DIV(w6b, maxF_nn(f.lu, zl));
          edx[is] = f.du * d;
          edy[is] = f.dv * d;
          if (le_nn(f.lu, zl) || geF(zl, w6b) || le_nn(w7sq, zl * zl) || le_nn(f.lx, zl)) {
            edx[is] = (lr)0;
            edy[is] = (lr)0;
          }
        }
      }
      const double visc = from_lr(vmax * DIV((lr)2, maxF(to_lr(rho0), zl)));
      F.cnviscx[iel] = make_d4(from_lr(edx[0] - edx[3]), from_lr(edx[1] - edx[0]),
                               from_lr(edx[2] - edx[1]), from_lr(edx[3] - edx[2]));
      F.cnviscy[iel] = make_d4(from_lr(edy[0] - edy[3]), from_lr(edy[1] - edy[0]),
                               from_lr(edy[2] - edy[1]), from_lr(edy[3] - edy[2]));
      F.visc[iel] = visc;
    }
  }
}

// ================================================================ k_getdt

// The mixed build's CFL and divergence candidates and the dt reduction, one
// thread per element.  Bound by its loads' latency (4 FP64 instructions an
// element): the positions are brought only for the regions and faces that
// need them, and a block takes several tiles.  (8, 10 and 12 blocks per SM,
// with the registers that leaves, are slower.)
template <int BS, bool BATCH, bool POS>
__global__ void __launch_bounds__(BS, BL_GETDT_MINB) k_getdt(DevFields F, DevCfg C) {
  DevStep* S = F.step;
  int blk0 = 0, nblk = (int)gridDim.x, el0 = 0, el1 = F.nel;
  const DevInst* I = nullptr;
  if (BATCH) {
    const int m = __ldg(F.blkinst + blockIdx.x);
    I = F.inst + m;
    S = F.steps + m;
    blk0 = I->blk_begin;
    nblk = I->blk_end - I->blk_begin;
    el0 = I->el_begin;
    el1 = I->el_end;
  }
  if (halted(S)) return;
  if (S->stop_next) {            // bl_run: the previous step reached time_end
    if ((int)blockIdx.x == blk0 && threadIdx.x == 0) S->halted = 1;
    return;
  }
  double cflv = HUGE_VAL;        // sentinel above HUGE(1.0)
  int cfli = 0x7fffffff;
  double divv = DBL_MIN;         // TINY(1.0)
  int divi = -1;
  const int tiles = getdt_tiles(F.nel, BS);
  int iel = el0 + ((int)blockIdx.x - blk0) * tiles * BS + (int)threadIdx.x;
  for (int k = 0; k < tiles && iel < el1; k++, iel += BS) {
    const int4 nd = __ldg(F.ielnd + iel);
    const int n[4] = {nd.x, nd.y, nd.z, nd.w};
    double u[4], v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      u[j] = F.ndu[n[j]];
      v[j] = F.ndv[n[j]];
    }
    auto corners = [&](double* x, double* y) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        x[j] = F.ndx[n[j]];
        y[j] = F.ndy[n[j]];
      }
    };
    getdt_tail<DevLayout, POS>(F, C, iel, corners, u, v, F.visc[iel], cflv, cfli, divv, divi);
  }
  getdt_finish<BS, BATCH>(F, C, S, cflv, cfli, divv, divi, blk0, nblk, el0, I);
}


#else
// Two kernels.  k_edge computes every edge of the mesh once
// (bl_setup.cuh: its slots); k_getdt then takes each element's four edges
// and does what depends on the element.  The edge viscosity's limiter, edge
// coefficient and lengths are the same seen from either element of an edge;
// one kernel per element computed each twice, a thread's four faces one
// after another.  Sedov 512x512: 145 us in one kernel, 69.6 us in two (218
// FP64 instructions, 31 divides and 9 square roots an element against about
// 110, 7 and 4); a 16,000-element Sod tube, where the one-thread chain was
// all of it, 42 to 28 us.
// the limiter of two ratios (hydro_kn_edgeviscosity.f90:185-199)
__device__ __forceinline__ double limit2(double r1, double r2) {
  return maxF(0.0, minF(minF(minF(half(r1 + r2), twice(r1)), twice(r2)), 1.0));
}

// the codes of an edge's continuing faces (bl_setup.cuh)
constexpr int kEndMirror = -2, kEndAdjacent = -3;

// position and velocity differences along a face, or a wall's ratio
struct EndD {
  double dx, dy, du, dv;
};
__device__ __forceinline__ EndD node_diff(const DevFields& F, int a, int b) {
  EndD d;
  d.dx = F.ndx[b] - F.ndx[a];
  d.dy = F.ndy[b] - F.ndy[a];
  d.du = F.ndu[b] - F.ndu[a];
  d.dv = F.ndv[b] - F.ndv[a];
  return d;
}

// biased exponent of |x| within [1023 + lo, 1023 + hi]
__device__ __forceinline__ bool exp_in(double x, int lo, int hi) {
  const int e = (int)((unsigned long long)bits64(x) >> 52) & 0x7ff;
  return (unsigned)(e - (1023 + lo)) <= (unsigned)(hi - lo);
}
// The limiter as the reference forms it, with its cut-offs: unit vectors
// and one quotient per ratio.  Out of line: k_edge needs it only for
// operands outside the range its own form covers.
static __device__ __noinline__ double limiter_general(double du, double dv, double dx, double dy,
                                                      int c1, EndD d1, int c2, EndD d2, double zc) {
  const FaceQ f = face_q(du, dv, dx, dy, zc);
  const double r1 = c1 < 0 && c1 != kEndAdjacent ? (c1 == kEndMirror ? 1.0 : 0.0)
                                                 : nb_ratio(f, d1.dx, d1.dy, d1.du, d1.dv, zc);
  const double r2 = c2 < 0 && c2 != kEndAdjacent ? (c2 == kEndMirror ? 1.0 : 0.0)
                                                 : nb_ratio(f, d2.dx, d2.dy, d2.du, d2.dv, zc);
  return limit2(r1, r2);
}

// ================================================================ k_edge

// One thread per slot; a block of BS threads takes BS - 2 consecutive
// slots, its first and last threads hold the neighbours of those and only
// publish.  Every thread publishes its edge's differences; an edge takes a
// continuing face from the thread beside it where the table says that it is
// that slot's edge (on meshes numbered along mesh lines all but the walls
// and the irregular faces), and gathers it from the nodes otherwise.
//
// With D = (dx, dy) and U = (du, dv) of this edge and
// D', U' of a continuing one, the reference's ratio is, in real arithmetic
// and away from its cut-offs, r = (U'.U |D|^2) / (|U|^2 D'.D): no square
// root, no unit vector.  The two products U'.U and D'.D are the same for
// the neighbour that continues into this edge, so each thread forms those
// with the next slot and hands them on: four operations a slot for both
// ends.  The limiter max(0, min((r1 + r2)/2, 2 r1, 2 r2, 1)) is then one
// quotient over the common denominator, and none where it is 0 or 1.  It
// holds while the squares and products keep clear of the range's ends and
// of zerocut (tested on their exponents: lengths from 2^-40 to 2^40,
// velocity differences from 2^-80 to 2^80, zerocut at most 2^-132; the
// default is 1e-40); other operands take limiter_general, among them the
// edges whose velocity difference is at most zerocut: their force is cut,
// their viscosity is not.  An edge without a difference has neither and skips
// the rest, as whole warps of still fluid do.
// Per edge it leaves (du, dv, E, EL), E = edge coefficient / |U| (0 where
// the reference cuts the edge) and EL = edge coefficient * |U|, and |D|^2.
#ifndef BL_EDGE_MINB
#define BL_EDGE_MINB 8
#endif
template <int BS, bool BATCH>
__global__ void __launch_bounds__(BS, BL_EDGE_MINB) k_edge(DevFields F, DevCfg C) {
  const int t = threadIdx.x;
  const int slot = (int)blockIdx.x * (BS - 2) + t - 1;
  bool in = slot >= 0 && slot < F.nslot;
  int4 n = make_int4(0, 0, 0, 0), q = make_int4(-1, -1, -1, -1);
  if (in) {
    n = __ldg(F.es_n + slot);
    q = __ldg(F.es_q + slot);
    if (BATCH) {
      const DevStep* S = el_step<true>(F, n.z);
      in = !(halted(S) || S->stop_next);
    }
  }
  if (!BATCH && (halted(F.step) || F.step->stop_next)) return;
  __shared__ double s_d[4][BS];
  EndD d = {0.0, 0.0, 0.0, 0.0};
  if (in) d = node_diff(F, n.x, n.y);
  s_d[0][t] = d.dx;
  s_d[1][t] = d.dy;
  s_d[2][t] = d.du;
  s_d[3][t] = d.dv;
  __syncthreads();
  const double zc = C.zerocut;
  auto diff = [&](int code, int node, int beside) {  // a continuing face's differences
    EndD r;
    if (code == kEndAdjacent) {
      r.dx = s_d[0][beside];
      r.dy = s_d[1][beside];
      r.du = s_d[2][beside];
      r.dv = s_d[3][beside];
    } else {
      r = node_diff(F, code, node);
    }
    return r;
  };
  __shared__ double s_p[BS], s_q[BS];
  if (t < BS - 1) {
    s_p[t] = fma(d.dv, s_d[3][t + 1], d.du * s_d[2][t + 1]);
    s_q[t] = fma(d.dy, s_d[1][t + 1], d.dx * s_d[0][t + 1]);
  }
  __syncthreads();
  if (!(in && t > 0 && t < BS - 1)) return;
  const double squ = fma(d.dv, d.dv, d.du * d.du), sqx = fma(d.dy, d.dy, d.dx * d.dx);
  double E = 0.0, EL = 0.0;
  if (!C.ztq && (bits64(squ) << 1) != 0) {
    const double lu = SQRT(squ);
    const double cs = SQRT(half(F.cs2[n.z] + F.cs2[n.w]));
    auto dots = [&](int code, int node, int beside, double& P, double& Q) {
      if (code == kEndAdjacent) {
        const int k = beside < t ? beside : t;
        P = s_p[k];
        Q = s_q[k];
      } else if (code < 0) {  // a wall's ratio 0, a mirrored face's 1
        P = code == kEndMirror ? squ : 0.0;
        Q = sqx;
      } else {
        const EndD o = node_diff(F, code, node);
        P = fma(d.dv, o.dv, d.du * o.du);
        Q = fma(d.dy, o.dy, d.dx * o.dx);
      }
    };
    double P1, Q1, P2, Q2, lim;
    dots(q.x, q.y, t - 1, P1, Q1);
    dots(q.z, q.w, t + 1, P2, Q2);
    bool cut = false;
    if (zc <= 0x1p-132 && exp_in(squ, -160, 160) && exp_in(sqx, -80, 80) &&
        exp_in(Q1, -80, 80) && exp_in(Q2, -80, 80) && exp_in(P1, -1023, 300) &&
        exp_in(P2, -1023, 300)) {
      const double QQ = Q1 * Q2;
      const double S1 = xorsign(P1 * Q2, QQ), S2 = xorsign(P2 * Q1, QQ);
      const double m = minF(minF(half(S1 + S2), twice(S1)), twice(S2));
      const double num = m * sqx, den = absF(QQ) * squ;
      lim = gtF(num, 0.0) ? (gtF(den, num) ? DIV(num, den) : 1.0) : 0.0;
    } else {
      const EndD none = {0.0, 0.0, 0.0, 0.0};
      const EndD o1 = q.x >= 0 || q.x == kEndAdjacent ? diff(q.x, q.y, t - 1) : none;
      const EndD o2 = q.z >= 0 || q.z == kEndAdjacent ? diff(q.z, q.w, t + 1) : none;
      lim = limiter_general(d.du, d.dv, d.dx, d.dy, q.x, o1, q.z, o2, zc);
      cut = le_nn(lu, zc) || le_nn(SQRT(sqx), zc);
    }
    const double edv = half(1.0 - lim) *
                       ((F.rho[n.z] + F.rho[n.w]) * fma(C.cvisc2, lu, C.cvisc1 * cs));
    EL = edv * lu;
    E = cut ? 0.0 : DIV(edv, lu);
  }
  F.erec[slot] = make_d4(d.du, d.dv, E, EL);
  F.esqx[slot] = sqx;
}

// ================================================================ k_getdt

// The element's CFL candidate over its squared signal speed cs2v, and its
// divergence candidate, from its coefficients and its edges' velocity
// differences and squared lengths (exact in real arithmetic):
// - with T1 = a1 b2 - a2 b1, T3 = a3 b2 - a2 b3 and the quarter volume
//   cross = a1 b3 - a3 b1, half the cross product of face f with the vector
//   from its midpoint to the centroid is W = cross + T3, cross + T1,
//   cross - T3, cross - T1; the reference's squared distance over squared
//   length of the side across face f (geometry_kn_dln) is 16 W^2 / |D|^2;
// - sum u_j (coefficient) is b1 (du3 - du1) + b3 (du0 - du2)
//   - a1 (dv3 - dv1) - a3 (dv0 - dv2).
__device__ __forceinline__ double cfl_candidate(const DevFields& F, const DevCfg& C, int iel,
                                                const double* W, const double* sq, double a1,
                                                double a2, double a3, double b1, double b2,
                                                double b3, double cs2v, int notdt, int mid) {
  if (notdt) return DBL_MAX;
  if (mid) {  // min over sides of |midpoint difference|^2
    const double r0 = a3 * a3 + b3 * b3, r1 = a1 * a1 + b1 * b1;
    return DIV(times4(minF_nn(r0, r1)), cs2v);
  }
  bool plain = true;
#pragma unroll
  for (int f = 0; f < 4; f++) plain = plain && !gt_nn(C.zcut, sq[f]) && exp_in(sq[f], -160, 160);
  if (plain) {
    // the smallest quotient by cross-multiplication: two products in place
    // of a divide
    double n = W[0] * W[0], d = sq[0];
#pragma unroll
    for (int f = 1; f < 4; f++) {
      const double nf = W[f] * W[f];
      if (gt_nn(n * sq[f], nf * d)) {
        n = nf;
        d = sq[f];
      }
    }
    return DIV(ldexpF<4>(n), d * cs2v);
  }
  // a face shorter than sqrt(zcut) counts with the distance from the
  // opposite midpoint to its first corner
  const double cx[4] = {a3, -a1, -a3, a1}, cy[4] = {b3, -b1, -b3, b1};
  const double hx[4] = {a1 - a2, a2 + a3, -(a1 + a2), a2 - a3};
  const double hy[4] = {b1 - b2, b2 + b3, -(b1 + b2), b2 - b3};
  double m = HUGE_VAL;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    double r;
    if (gt_nn(C.zcut, sq[f])) {
      const double x = twice(cx[f]) + hx[f], y = twice(cy[f]) + hy[f];
      r = x * x + y * y;
    } else {
      r = DIV(ldexpF<4>(W[f] * W[f]), sq[f]);
    }
    m = minF_nn(m, r);
  }
  return DIV(m, cs2v);
}

// One thread per element: its corner viscosity forces and viscosity from
// its edges, elcs2 + elvisc, and its CFL and divergence candidates; then
// the dt reduction.  (POS: DevFields::geom_x)
template <int BS, bool BATCH, bool POS>
__global__ void __launch_bounds__(BS, BL_GETDT_MINB) k_getdt(DevFields F, DevCfg C) {
  // the mesh of this block: the context's, or in a batch the block's own
  // (its blocks [blk0, blk0 + nblk), elements [el0, el1))
  DevStep* S = F.step;
  int blk0 = 0, nblk = (int)gridDim.x, el0 = 0, el1 = F.nel;
  const DevInst* I = nullptr;
  if (BATCH) {
    const int m = __ldg(F.blkinst + blockIdx.x);
    I = F.inst + m;
    S = F.steps + m;
    blk0 = I->blk_begin;
    nblk = I->blk_end - I->blk_begin;
    el0 = I->el_begin;
    el1 = I->el_end;
  }
  const int tiles = getdt_tiles(F.nel, BS);
  int iel = el0 + ((int)blockIdx.x - blk0) * tiles * BS + (int)threadIdx.x;
  // (the table's load leaves before the header's answer is needed)
  uint4 er4 = make_uint4(0u, 0u, 0u, 0u);
  if (iel < el1) er4 = __ldg(F.eref + iel);
  if (halted(S)) return;
  if (S->stop_next) {            // bl_run: the previous step reached time_end
    if ((int)blockIdx.x == blk0 && threadIdx.x == 0) S->halted = 1;
    return;
  }
  double cflv = HUGE_VAL;        // sentinel above HUGE(1.0)
  int cfli = 0x7fffffff;
  double divv = DBL_MIN;         // TINY(1.0)
  int divi = -1;
  for (int k = 0; k < tiles && iel < el1; k++, iel += BS) {
    if (k > 0) er4 = __ldg(F.eref + iel);
    const unsigned er[4] = {er4.x, er4.y, er4.z, er4.w};
    double visc = 0.0;
    double du[4], dv[4], sq[4], W[4], edx[4], edy[4];
    double a1 = F.a1[iel], a2, a3 = F.a3[iel], b1 = F.b1[iel], b2, b3 = F.b3[iel];
    const double vol = F.vol[iel], rho = F.rho[iel], cs2 = F.cs2[iel];
    // the divergence limit's coefficients are the stored ones in any case
    const double da1 = a1, da3 = a3, db1 = b1, db3 = b3;
    const int ireg = __ldg(F.ielreg + iel);
    const int notdt = __ldg(C.zdtnotreg + ireg), mid = __ldg(C.zmidlength + ireg);
    {
      double cross;
      if (POS) {
        const int4 n = __ldg(F.ielnd + iel);
        const double x[4] = {F.ndx[n.x], F.ndx[n.y], F.ndx[n.z], F.ndx[n.w]};
        const double y[4] = {F.ndy[n.x], F.ndy[n.y], F.ndy[n.z], F.ndy[n.w]};
        const Iso g = getiso(x, y);
        a1 = g.a1, a2 = g.a2, a3 = g.a3, b1 = g.b1, b2 = g.b2, b3 = g.b3;
        cross = g.cross;
      } else {
        a2 = F.a2[iel];
        b2 = F.b2[iel];
        cross = quarter(vol);
      }
      const double t1 = a1 * b2 - a2 * b1, t3 = a3 * b2 - a2 * b3;
      W[0] = cross + t3;
      W[1] = cross + t1;
      W[2] = cross - t3;
      W[3] = cross - t1;
    }
    const double zc = C.zerocut;
    // |midpoint to centroid| above zerocut: (a3,b3) for faces 0 and 2,
    // (a1,b1) for 1 and 3 (a component above it says so without the square)
    const bool cut0 = !(gt_nn(absF(a3), zc) || gt_nn(absF(b3), zc)) && le_nn(a3 * a3 + b3 * b3, zc * zc);
    const bool cut1 = !(gt_nn(absF(a1), zc) || gt_nn(absF(b1), zc)) && le_nn(a1 * a1 + b1 * b1, zc * zc);
    double vmax = 0.0;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const unsigned slot = er[f] >> 1;
      const d4 R = F.erec[slot];
      sq[f] = F.esqx[slot];
      const double sg = from_bits64((long long)((unsigned long long)(er[f] & 1u) << 63));
      du[f] = xorsign(R.x, sg);
      dv[f] = xorsign(R.y, sg);
      vmax = maxF_nn(vmax, R.w);  // never negative
      // edge force (hydro_kn_edgeviscosity.f90:219-282): the reference
      // normalises the midpoint-to-centroid vector c, orients it by the
      // sign of its product with the face vector (that of W) and scales it
      // back by |c|; so the force is U E times -+(U x c)
      const double cx = (f & 1) ? a1 : a3, cy = (f & 1) ? b1 : b3;
      const double g = dv[f] * cx - du[f] * cy;  // c has the other sign for faces 1 and 2
      const double w6 = (f == 1 || f == 2) ? negxorsign(g, W[f]) : xorsign(g, W[f]);
      const double d = R.z * w6;
      const bool cut = geF(zc, w6) || ((f & 1) ? cut1 : cut0);
      edx[f] = cut ? 0.0 : du[f] * d;
      edy[f] = cut ? 0.0 : dv[f] * d;
    }
    if (!C.ztq) {
      visc = DIV(twice(vmax), maxF(rho, zc));
      F.cnviscx[iel] = make_d4(edx[0] - edx[3], edx[1] - edx[0], edx[2] - edx[1], edx[3] - edx[2]);
      F.cnviscy[iel] = make_d4(edy[0] - edy[3], edy[1] - edy[0], edy[2] - edy[1], edy[3] - edy[2]);
      F.visc[iel] = visc;
    } else {
      visc = F.visc[iel];
    }
    const double cs2v = signal_speed(F, iel, cs2, visc);
    cfl_min(cflv, cfli, cfl_candidate(F, C, iel, W, sq, a1, a2, a3, b1, b2, b3, cs2v, notdt, mid),
            iel);
    const double w = db1 * (du[3] - du[1]) + db3 * (du[0] - du[2]) - da1 * (dv[3] - dv[1]) -
                     da3 * (dv[0] - dv[2]);
    const double dd = DIV(absF(w), vol);
    if (gt_nn(dd, divv)) {
      divv = dd;
      divi = iel;
    }
  }
  getdt_finish<BS, BATCH>(F, C, S, cflv, cfli, divv, divi, blk0, nblk, el0, I);
}

#endif
#else

// ================================================================ k_edge

// Exact build: the edge viscosity, one thread per face of an element, four
// adjacent threads an element.  Both elements of an edge compute it, each in
// its own order (a reversed difference can differ from the recomputed one in
// the sign of a zero), and every expression is the reference's; the quad
// joins its faces through shuffles.  One thread per element took its four
// faces one after another with 676 bytes of spills; the step of a 1,000-element
// tube took 66.9 us, now 41.6, Sedov 128x128 89.8, now 68.5, 512x512 596, now 581.
// An edge whose ends move alike -- fluid at rest -- has length 0 in velocity:
// whatever the limiter says its force is cut (0 <= zerocut) and its viscosity
// is 0 (or 0 in MAX's first place against a NaN), so it stops there:
// Sedov 512x512
// after 60 steps 556 -> 395 us a step, 128x128 67.9 -> 63.9.
#ifndef BL_EDGE_MINB
#define BL_EDGE_MINB 7
#endif
template <int BS, bool BATCH, class L = DevLayout>
__global__ void __launch_bounds__(BS, BL_EDGE_MINB) k_edge(DevFields F, DevCfg C) {
  const long long at = (long long)blockIdx.x * BS + threadIdx.x;
  const int iel = (int)(at >> 2), is = (int)(at & 3), jn = (is + 1) & 3;
  bool in = iel < F.nel;  // the same for a quad
  if (!BATCH && (halted(F.step) || F.step->stop_next)) return;
  if (BATCH && in) {
    const DevStep* S = el_step<true>(F, iel);
    in = !(halted(S) || S->stop_next);
  }
  auto ipick = [](const int4& v, int j) {
    return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
  };
  double ex = 0.0, ey = 0.0, visc = 0.0;
  double du = 0.0, dv = 0.0, squ = 0.0;
  int4 n = make_int4(0, 0, 0, 0);
  if (in) {
    n = L::nodes(F, iel);
    const int na = ipick(n, is), nn = ipick(n, jn);
    du = F.ndu[nn] - F.ndu[na];
    dv = F.ndv[nn] - F.ndv[na];
    squ = du * du + dv * dv;
  }
  if (in && ((bits64(squ) << 1) != 0 || !geF(C.zerocut, 0.0))) {
    // hydro_kn_initeviscosity / limiteviscosity / geteviscosity
    // (hydro_kn_edgeviscosity.f90:30-282).  Face is runs corner is -> is+1;
    // the faces of side s (neighbours across faces s and s+2) are (s+3)&3
    // and s+1.
    const int4 nb = L::nbrs(F, iel);
    const int fcp = L::faces(F, iel);
    const double zc = C.zerocut;
    const double rho0 = F.rho[iel], cs2i = F.cs2[iel];
    const double x[4] = {F.ndx[n.x], F.ndx[n.y], F.ndx[n.z], F.ndx[n.w]};
    const double y[4] = {F.ndy[n.x], F.ndy[n.y], F.ndy[n.z], F.ndy[n.w]};
    const double xc = quarter(x[0] + x[1] + x[2] + x[3]);
    const double yc = quarter(y[0] + y[1] + y[2] + y[3]);
    auto pick = [](const double* v, int j) {
      return j == 0 ? v[0] : (j == 1 ? v[1] : (j == 2 ? v[2] : v[3]));
    };
    const double xa = pick(x, is), xb = pick(x, jn), ya = pick(y, is), yb = pick(y, jn);
    const int s = (is & 1) ? 0 : 1;
    const bool first = is == 3 || is == 0;
    const int in1 = ipick(nb, s), in2 = ipick(nb, s + 2);
    const int f1 = fc_of(fcp, s), f2 = fc_of(fcp, s + 2);
    // boundary rule (hydro_kn_edgeviscosity.f90:154-183): a ratio across a
    // boundary face is 1 between two boundary nodes facing an interior
    // neighbour, 0 otherwise
    double r1 = 0.0, r2 = 0.0;
    if (in1 == iel)
      r1 = (__ldg(F.indtype + ipick(n, s)) < 0 && __ldg(F.indtype + ipick(n, s + 1)) < 0 &&
            in2 != iel) ? 1.0 : 0.0;
    if (in2 == iel)
      r2 = (__ldg(F.indtype + ipick(n, s + 2)) < 0 &&
            __ldg(F.indtype + ipick(n, (s + 3) & 3)) < 0 && in1 != iel) ? 1.0 : 0.0;
    double w1 = du, w2 = dv;
    double w3 = xb - xa, w4 = yb - ya;
    double den = SQRT(squ);
    const double lu = den;
    den = DIV(1.0, maxF_nn(den, zc));
    const double uhat = w1 * den, vhat = w2 * den;
    den = SQRT(w3 * w3 + w4 * w4);
    const double lx = den;
    den = DIV(1.0, maxF_nn(den, zc));
    const double xh = w3 * den, yh = w4 * den;
    den = w3 * xh + w4 * yh;
    w1 = DIV(w1 * uhat + w2 * vhat, signF(maxF_nn(absF(den), zc), den));
    w1 = DIV(1.0, signF(maxF_nn(absF(w1), zc), w1));
    // neighbour faces: edge 1 uses MOD(ielfc,4)+1 / MOD(ielfc+2,4)+1,
    // edge 2 the other pair (hydro_kn_edgeviscosity.f90:117-151)
    auto ratio = [&](int nbr, int face) {
      const int4 m = L::nodes(F, nbr);
      const int a = ipick(m, face), b = ipick(m, (face + 1) & 3);
      const double ddx = F.ndx[b] - F.ndx[a], ddy = F.ndy[b] - F.ndy[a];
      const double ddu = F.ndu[b] - F.ndu[a], ddv = F.ndv[b] - F.ndv[a];
      const double dn = ddx * xh + ddy * yh;
      const double q = DIV(ddu * uhat + ddv * vhat, signF(maxF_nn(absF(dn), zc), dn));
      return q * w1;
    };
    if (in1 != iel) r1 = ratio(in1, (f1 + (first ? 1 : 3)) & 3);
    if (in2 != iel) r2 = ratio(in2, (f2 + (first ? 3 : 1)) & 3);
    // limiter and edge coefficient (hydro_kn_edgeviscosity.f90:185-214)
    const int ins = ipick(nb, is);
    w1 = C.cvisc1 * SQRT(half(cs2i + F.cs2[ins]));
    w2 = minF(minF(minF(half(r1 + r2), twice(r1)), twice(r2)), 1.0);
    w2 = maxF(0.0, w2);
    w3 = half(1.0 - w2) * (rho0 + F.rho[ins]) * (w1 + C.cvisc2 * lu);
    const double edv = w3;
    visc = maxF_nn(0.0, w3 * DIV(twice(lu), maxF(rho0, zc)));
    // edge force (hydro_kn_edgeviscosity.f90:219-282)
    const double m3 = half(xa + xb);
    const double m6 = half(ya + yb);
    const double w7 = SQRT((xc - m3) * (xc - m3) + (yc - m6) * (yc - m6));
    double d = DIV(1.0, w7);
    double exh = (yc - m6) * d, eyh = (m3 - xc) * d;
    // w1*(1/w8), w4*(1/w8) with w8 the face's length: the limiter's
    // normalised face vector whenever w8 > zerocut; otherwise the edge is
    // cut below
    const double w33 = exh * xh + eyh * yh;
    d = -(signF(1.0, w33) * w7);
    exh = exh * d;
    eyh = eyh * d;
    const double w6b = du * exh + dv * eyh;
    d = DIV(w6b, maxF_nn(lu, zc));
    if (!(le_nn(lu, zc) || geF(zc, w6b) || le_nn(w7, zc) || le_nn(lx, zc))) {
      ex = edv * du * d;
      ey = edv * dv * d;
    }
  }
  // corner j's force is the difference of faces j and j - 1; elvisc is the
  // largest of the four faces' (never negative: +0 or positive)
  const int from = (threadIdx.x & 28) | ((is + 3) & 3);
  const double px = __shfl_sync(0xffffffffu, ex, from), py = __shfl_sync(0xffffffffu, ey, from);
  visc = maxF_nn(visc, __shfl_xor_sync(0xffffffffu, visc, 1));
  visc = maxF_nn(visc, __shfl_xor_sync(0xffffffffu, visc, 2));
  if (in) {
    reinterpret_cast<double*>(F.cnviscx)[at] = ex - px;
    reinterpret_cast<double*>(F.cnviscy)[at] = ey - py;
    if (is == 0) F.visc[iel] = visc;
  }
}

// ================================================================ k_getdt

// Exact build: hydro_dr_getcs2, the CFL and divergence candidates and the dt
// reduction, after k_edge.
template <int BS, bool BATCH, class L = DevLayout>
__global__ void __launch_bounds__(BS, BL_GETDT_MINB) k_getdt(DevFields F, DevCfg C) {
  // the mesh of this block: the context's, or in a batch the block's own
  // (its blocks [blk0, blk0 + nblk), elements [el0, el1))
  DevStep* S = F.step;
  int blk0 = 0, nblk = (int)gridDim.x, el0 = 0, el1 = F.nel;
  const DevInst* I = nullptr;
  if (BATCH) {
    const int m = __ldg(F.blkinst + blockIdx.x);
    I = F.inst + m;
    S = F.steps + m;
    blk0 = I->blk_begin;
    nblk = I->blk_end - I->blk_begin;
    el0 = I->el_begin;
    el1 = I->el_end;
  }
  if (halted(S)) return;
  if (S->stop_next) {            // bl_run: the previous step reached time_end
    if ((int)blockIdx.x == blk0 && threadIdx.x == 0) S->halted = 1;
    return;
  }
  const int iel = el0 + ((int)blockIdx.x - blk0) * BS + threadIdx.x;
  double cflv = HUGE_VAL;        // sentinel above HUGE(1.0)
  int cfli = 0x7fffffff;
  double divv = DBL_MIN;         // TINY(1.0)
  int divi = -1;
  if (iel < el1) {
    const int4 nd = L::nodes(F, iel);
    const int n[4] = {nd.x, nd.y, nd.z, nd.w};
    double u[4], v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      u[j] = F.ndu[n[j]];
      v[j] = F.ndv[n[j]];
    }
    auto corners = [&](double* x, double* y) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        x[j] = F.ndx[n[j]];
        y[j] = F.ndy[n[j]];
      }
    };
    getdt_tail<L>(F, C, iel, corners, u, v, F.visc[iel], cflv, cfli, divv, divi);
  }
  getdt_finish<BS, BATCH>(F, C, S, cflv, cfli, divv, divi, blk0, nblk, el0, I);
}
#endif

// ================================================================ k_lag_force

#if BL_FAST_ALGEBRA
// Fast build.  Only the energy needs the predictor's forces, and only their
// work sum f_j . u_j, so that is formed directly; the half-step geometry
// follows from the element's own coefficients, which are linear in the
// corner positions; the corrector's pressure, sub-zonal and hourglass forces
// share their sums.  (All exact in real arithmetic.)  With
//   d = (b1 - b3), s = (b1 + b3), U02 = u0 - u2, U13 = u1 - u3,
//   h = u0 - u1 + u2 - u3 (and the same with a and v for y, sign reversed):
// - pressure work: p Dv, Dv = d U02 + s U13 - (y);
// - a1, a2, a3 at the half step: a1 + dt/8 (U13 - U02), a2 + dt/8 h,
//   a3 - dt/8 (U02 + U13);
// - sub-zonal pressures (hydro_kn_getforce.f90:109-188): the sub-quad of
//   corner j has the volume V_j = cross + td/2, cross + ts/2, cross - td/2,
//   cross - ts/2 (cross = a1 b3 - a3 b1, ts = T1 + T3, td = T3 - T1,
//   T1 = a1 b2 - a2 b1, T3 = a3 b2 - a2 b3) and the pressure p_j = cs2
//   (spmass_j / V_j - rho); in the reference's gather of the sub-quads'
//   forces to the corners the midpoint terms of adjacent ones cancel
//   pairwise.  With P_j = pmerit p_j / 2, S02 = P0 + P2, M02 = P0 - P2 (S13,
//   M13 likewise), the corner x forces are
//     f0 =  d P0 + D13 - G, f2 = -d P2 - D13 - G,
//     f1 =  s P1 + D02 - G, f3 = -s P3 - D02 - G,
//     D13 = (d S13 - b2 M13)/2, D02 = (s S02 - b2 M02)/2,
//     G = (d M02 + s M13)/4,
//   and their work, with q_j = spmass_j / V_j,
//     pmerit cs2 / 8 (2 Dv (sum q_j - 4 rho) + B (q0 - q2) - C (q1 - q3)),
//     B = d h - 2 b2 U13 - (y), C = s h + 2 b2 U02 - (y).
// 152 FP64 instructions an element in motion with all forces on where the
// reference's terms one by one took 206, and no corner positions gathered:
// Sedov 512x512 108 -> 88 us, 42 -> 39 us at 90,000 elements; FP64 pipe 71 %
// busy over the SMs' active cycles, the divide chains' latency the rest (blocks
// and bound: BL_FORCE_MINB).
// POS: where the coefficients or volumes are not those of the positions
// (DevFields::geom_x), the half-step geometry and the sub-zonal pressures are
// formed from the corners; the pressure force keeps the stored coefficients,
// as the reference's does.
struct SubZone {
  double q[4];  // sub-zonal densities spmass_j / V_j
};
__device__ __forceinline__ SubZone sub_zone(double cross, double ts, double td, const d4& spm) {
  SubZone z;
  z.q[0] = DIV_IN(spm.x, fma(td, 0.5, cross));
  z.q[1] = DIV_IN(spm.y, fma(ts, 0.5, cross));
  z.q[2] = DIV_IN(spm.z, fma(-td, 0.5, cross));
  z.q[3] = DIV_IN(spm.w, fma(-ts, 0.5, cross));
  return z;
}
// one direction's corner forces (sg = 1: x from the b's, -1: y from the
// a's); w the hourglass force of the even corners
template <int SG>
__device__ __forceinline__ void corner_forces(double d, double s, double c2, const double* P,
                                              double S02, double M02, double S13, double M13,
                                              double w, const d4& q, double* f) {
  const double G = quarter(fma(d, M02, s * M13));
  const double D13 = half(fma(d, S13, -(c2 * M13))), D02 = half(fma(s, S02, -(c2 * M02)));
  if (SG > 0) {
    const double e = w - G, o = -w - G;
    f[0] = fma(d, P[0], (e + D13) + q.x);
    f[1] = fma(s, P[1], (o + D02) + q.y);
    f[2] = fma(-d, P[2], (e - D13) + q.z);
    f[3] = fma(-s, P[3], (o - D02) + q.w);
  } else {
    const double e = w + G, o = G - w;
    f[0] = fma(-d, P[0], (e - D13) + q.x);
    f[1] = fma(-s, P[1], (o - D02) + q.y);
    f[2] = fma(d, P[2], (e + D13) + q.z);
    f[3] = fma(s, P[3], (o + D02) + q.w);
  }
}

template <int BS, bool BATCH, bool POS>
__global__ void __launch_bounds__(BS, BL_FORCE_MINB) k_lag_force(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  const int4 nd = __ldg(F.ielnd + iel);
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted(S)) return;
  const double dt = S->dt;
  const double hdt = half(dt);   // time_dr_setpredictor dts / getvertex step
  const double zc = C.zerocut;
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  double u[4], v[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    u[j] = F.ndu[n[j]];
    v[j] = F.ndv[n[j]];
  }
  const d4 qx = F.cnviscx[iel], qy = F.cnviscy[iel];
  const int ireg = __ldg(F.ielreg + iel);
  const EosTab mat = eos_tab(C, __ldg(F.ielmat + iel));
  const double m = F.mass[iel];
  const double e0 = F.e[iel];
  const int imx = F.elmx ? F.elmx[iel] : -1;
  const double a1 = F.a1[iel], a2 = F.a2[iel], a3 = F.a3[iel];
  const double b1 = F.b1[iel], b2 = F.b2[iel], b3 = F.b3[iel];
  const double pm = C.zsp ? __ldg(C.pmeritreg + ireg) : 0.0;
  const double p0 = F.p[iel];
  // ---- the predictor forces' work at t^n (hydro_dr_getforce, zcorrector false):
  // none on fluid at rest, with finite forces (a third of the kernel's FP64
  // instructions with the sub-zonal pressure: Sedov 512x512 after 60 steps
  // 87.5 -> 61.8 us, Noh 1024x1024, all in motion, 143.7 and 143.7)
  double u02 = 0.0, u13 = 0.0, v02 = 0.0, v13 = 0.0, hu = 0.0, hv = 0.0, work = 0.0;
  long long still = bits64(u[0]) | bits64(u[1]) | bits64(u[2]) | bits64(u[3]) | bits64(v[0]) |
                    bits64(v[1]) | bits64(v[2]) | bits64(v[3]);
  bool rest = (still << 1) == 0;
  if (rest) {
    unsigned x = 0;
    for (const double f : {p0, a1, a2, a3, b1, b2, b3, qx.x, qx.y, qx.z, qx.w, qy.x, qy.y, qy.z,
                           qy.w, e0})
      x = max(x, (unsigned)(bits64(f) >> 32) & 0x7ff00000u);
    if (C.zsp)
      for (const double f : {F.vol[iel], F.rho[iel], F.cs2v[iel]})
        x = max(x, (unsigned)(bits64(f) >> 32) & 0x7ff00000u);
    rest = x != 0x7ff00000u;
  }
  if (!rest) {
    u02 = u[0] - u[2];
    u13 = u[1] - u[3];
    v02 = v[0] - v[2];
    v13 = v[1] - v[3];
    hu = (u[0] + u[2]) - (u[1] + u[3]);
    hv = (v[0] + v[2]) - (v[1] + v[3]);
    const double d = b1 - b3, s = b1 + b3, dy = a1 - a3, sy = a1 + a3;
    const double Dv = (d * u02 + s * u13) - (dy * v02 + sy * v13);
    work = p0 * Dv + qx.x * u[0] + qy.x * v[0] + qx.y * u[1] + qy.y * v[1] + qx.z * u[2] +
           qy.z * v[2] + qx.w * u[3] + qy.w * v[3];
    auto sub_zone_work = [&](const SubZone& z, double d, double s, double dy, double sy, double a2,
                             double b2, double Dv) {
      const double b22 = twice(b2), a22 = twice(a2);
      const double B = (d * hu - b22 * u13) - (dy * hv - a22 * v13);
      const double D = (s * hu + b22 * u02) - (sy * hv + a22 * v02);
      const double sum = fma(-4.0, F.rho[iel], (z.q[0] + z.q[2]) + (z.q[1] + z.q[3]));
      const double w = fma(twice(Dv), sum, fma(B, z.q[0] - z.q[2], -(D * (z.q[1] - z.q[3]))));
      return fma(ldexpF<-3>(pm) * F.cs2v[iel], w, work);
    };
    if (C.zsp && !POS) {
      const double t1 = a1 * b2 - a2 * b1, t3 = a3 * b2 - a2 * b3;
      const SubZone z = sub_zone(quarter(F.vol[iel]), t1 + t3, t3 - t1, F.spmass[iel]);
      work = sub_zone_work(z, d, s, dy, sy, a2, b2, Dv);
    } else if (C.zsp) {
      double x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        x[j] = F.ndx[n[j]];
        y[j] = F.ndy[n[j]];
      }
      const Iso g = getiso(x, y);
      const SubZone z = sub_zone(g.cross, g.ts, g.td, F.spmass[iel]);
      const double gd = g.b1 - g.b3, gs = g.b1 + g.b3, gdy = g.a1 - g.a3, gsy = g.a1 + g.a3;
      work = sub_zone_work(z, gd, gs, gdy, gsy, g.a2, g.b2,
                           (gd * u02 + gs * u13) - (gdy * v02 + gsy * v13));
    }
  }
  // ---- geometry at the half step (geometry_kn_getvertex with 0.5*dt,
  // geometry_dr_getgeometry), density
  Iso g;
  if (!POS) {
    const double r = quarter(hdt);
    g.a1 = fma(r, u13 - u02, a1);
    g.a2 = fma(r, hu, a2);
    g.a3 = fma(-r, u02 + u13, a3);
    g.b1 = fma(r, v13 - v02, b1);
    g.b2 = fma(r, hv, b2);
    g.b3 = fma(-r, v02 + v13, b3);
    iso_volumes(g);
  } else {
    double xh[4], yh[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      xh[j] = F.ndx[n[j]] + hdt * u[j];
      yh[j] = F.ndy[n[j]] + hdt * v[j];
    }
    g = getiso(xh, yh);
  }
  if (gtF(0.0, g.vol)) note_negvol(F, S, &DevStep::negvol_pred, iel + 1 - el_base<BATCH>(F, iel));
  const double rho = DIV_IN(m, g.vol);
  // ---- energy (hydro_kn_getenergy with dts = dt/2) and EoS
  const double eh = e0 - DIV_IN(work, maxF(m, zc)) * hdt;
  double ph, cs2h;
  eos_pc(C, mat, rho, eh, ph, cs2h);
  double fx[4], fy[4];
  // ---- mixed cells: component state at the half step
  if (imx >= 0) {
    const int c0 = F.imxfcp[imx], nc = F.imxncp[imx];
    if (F.closure && nc == 2) F.mxv0[imx] = F.vol[iel];  // for k_mix_closure
    double ax[4] = {0, 0, 0, 0}, ay[4] = {0, 0, 0, 0};
    for (int k = 0; k < nc; k++) {
      const int icp = c0 + k;
      const double fr = F.frvol[icp];
      // predictor component force with the t^n component state
      double cfx[4], cfy[4];
      force_pq(F.cpp[icp], a1, a3, b1, b3, F.cpviscx[icp],
               F.cpviscy[icp], cfx, cfy);
      // component energy with cpu = frvolume*cnu (utils_kn_mxgathercnav)
      double cu[4], cv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cu[j] = fr * u[j];
        cv[j] = fr * v[j];
      }
      const double cpm = F.cpm[icp];
      const double cpe = energy_update(F.cpe[icp], cpm, zc, hdt, cfx, cfy, cu, cv);
      F.cpe[icp] = cpe;  // the reference does not restore component energy
      const double cpv = times4(g.a1 * g.b3 - g.a3 * g.b1) * fr;
      const double cpr = DIV(cpm, cpv);
      double cpp, cpc;
      eos_pc(C, __ldg(F.icpmat + icp), cpr, cpe, cpp, cpc);
      // corrector component force at the half-step state
      force_pq(cpp, g.a1, g.a3, g.b1, g.b3, F.cpviscx[icp], F.cpviscy[icp], cfx, cfy);
      F.cpfx[icp] = make_d4(cfx[0], cfx[1], cfx[2], cfx[3]);
      F.cpfy[icp] = make_d4(cfy[0], cfy[1], cfy[2], cfy[3]);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        ax[j] = ax[j] + fr * cfx[j];
        ay[j] = ay[j] + fr * cfy[j];
      }
    }
    // corrector element force: P+Q+SP+HG are overwritten by the average
#pragma unroll
    for (int j = 0; j < 4; j++) {
      fx[j] = ax[j];
      fy[j] = ay[j];
    }
  } else {
    // ---- corrector force at the half step (zcorrector true)
    const double d = g.b1 - g.b3, s = g.b1 + g.b3, dy = g.a1 - g.a3, sy = g.a1 + g.a3;
    double wx = 0.0, wy = 0.0;
    if (C.zhg) {  // hydro_kn_getforceHG (hydro_kn_getforce.f90:73-107)
      const double w = -__ldg(C.kappareg + ireg) * rho * g.vol * S->rdt;
      wx = w * hu;
      wy = w * hv;
    }
    if (C.zsp) {
      const SubZone z = sub_zone(g.cross, g.ts, g.td, F.spmass[iel]);
      const double c = half(pm) * cs2h, cr = c * rho;
      double P[4];
#pragma unroll
      for (int j = 0; j < 4; j++) P[j] = fma(c, z.q[j], -cr);
      const double S02 = P[0] + P[2], M02 = P[0] - P[2], S13 = P[1] + P[3], M13 = P[1] - P[3];
#pragma unroll
      for (int j = 0; j < 4; j++) P[j] = P[j] + ph;
      corner_forces<1>(d, s, g.b2, P, S02, M02, S13, M13, wx, qx, fx);
      corner_forces<-1>(dy, sy, g.a2, P, S02, M02, S13, M13, wy, qy, fy);
    } else {
      fx[0] = fma(ph, d, qx.x);
      fx[1] = fma(ph, s, qx.y);
      fx[2] = fma(-ph, d, qx.z);
      fx[3] = fma(-ph, s, qx.w);
      fy[0] = fma(-ph, dy, qy.x);
      fy[1] = fma(-ph, sy, qy.y);
      fy[2] = fma(ph, dy, qy.z);
      fy[3] = fma(ph, sy, qy.w);
      if (C.zhg) {
        fx[0] += wx;
        fx[1] -= wx;
        fx[2] += wx;
        fx[3] -= wx;
        fy[0] += wy;
        fy[1] -= wy;
        fy[2] += wy;
        fy[3] -= wy;
      }
    }
  }
  F.cnfx[iel] = make_d4(fx[0], fx[1], fx[2], fx[3]);
  F.cnfy[iel] = make_d4(fy[0], fy[1], fy[2], fy[3]);
  F.rho_h[iel] = rho;
  F.cnwt_h[iel] = make_d4(g.w0, g.w1, g.w2, g.w3);
}
#else
template <int BS, bool BATCH>
__global__ void __launch_bounds__(BS, BL_FORCE_MINB) k_lag_force(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted(S)) return;
  const double dt = S->dt;
  const double hdt = 0.5 * dt;   // time_dr_setpredictor dts / getvertex step
  const double zc = C.zerocut;
  const int4 nd = __ldg(F.ielnd + iel);
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  double x[4], y[4], u[4], v[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    x[j] = F.ndx[n[j]];
    y[j] = F.ndy[n[j]];
    u[j] = F.ndu[n[j]];
    v[j] = F.ndv[n[j]];
  }
  const d4 qx = F.cnviscx[iel], qy = F.cnviscy[iel];
  const int ireg = __ldg(F.ielreg + iel);
  const int mat = __ldg(F.ielmat + iel);
  const double m = F.mass[iel];
  const double e0 = F.e[iel];
  const int imx = F.elmx ? F.elmx[iel] : -1;
  double fx[4], fy[4];
  // ---- predictor force at t^n (hydro_dr_getforce, zcorrector false)
  const double a1 = F.a1[iel], a3 = F.a3[iel], b1 = F.b1[iel], b3 = F.b3[iel];
  force_pq(F.p[iel], a1, a3, b1, b3, qx, qy, fx, fy);
  if (C.zsp) {
    force_sp(__ldg(C.pmeritreg + ireg), F.rho[iel], F.cs2v[iel], x, y, F.spmass[iel], fx, fy);
  }
  // ---- half-step vertices (geometry_kn_getvertex with 0.5*dt)
  double xh[4], yh[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    xh[j] = x[j] + hdt * u[j];
    yh[j] = y[j] + hdt * v[j];
  }
  // ---- geometry, density (geometry_dr_getgeometry, density_dr_getdensity)
  Iso g = getiso(xh, yh);
  if (gtF(0.0, g.vol)) note_negvol(F, S, &DevStep::negvol_pred, iel + 1 - el_base<BATCH>(F, iel));
  const double rho = DIV(m, g.vol);
  // ---- energy (hydro_kn_getenergy with dts = dt/2) and EoS
  const double eh = energy_update(e0, m, zc, hdt, fx, fy, u, v);
  double ph, cs2h;
  eos_pc(C, mat, rho, eh, ph, cs2h);
  // ---- mixed cells: component state at the half step
  if (imx >= 0) {
    const int c0 = F.imxfcp[imx], nc = F.imxncp[imx];
    if (F.closure && nc == 2) F.mxv0[imx] = F.vol[iel];  // for k_mix_closure
    double ax[4] = {0, 0, 0, 0}, ay[4] = {0, 0, 0, 0};
    for (int k = 0; k < nc; k++) {
      const int icp = c0 + k;
      const double fr = F.frvol[icp];
      // predictor component force with the t^n component state
      double cfx[4], cfy[4];
      force_pq(F.cpp[icp], a1, a3, b1, b3, F.cpviscx[icp],
               F.cpviscy[icp], cfx, cfy);
      // component energy with cpu = frvolume*cnu (utils_kn_mxgathercnav)
      double cu[4], cv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cu[j] = fr * u[j];
        cv[j] = fr * v[j];
      }
      const double cpm = F.cpm[icp];
      const double cpe = energy_update(F.cpe[icp], cpm, zc, hdt, cfx, cfy, cu, cv);
      F.cpe[icp] = cpe;  // the reference does not restore component energy
      const double cpv = times4(g.a1 * g.b3 - g.a3 * g.b1) * fr;
      const double cpr = DIV(cpm, cpv);
      double cpp, cpc;
      eos_pc(C, __ldg(F.icpmat + icp), cpr, cpe, cpp, cpc);
      // corrector component force at the half-step state
      force_pq(cpp, g.a1, g.a3, g.b1, g.b3, F.cpviscx[icp], F.cpviscy[icp], cfx, cfy);
      F.cpfx[icp] = make_d4(cfx[0], cfx[1], cfx[2], cfx[3]);
      F.cpfy[icp] = make_d4(cfy[0], cfy[1], cfy[2], cfy[3]);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        ax[j] = ax[j] + fr * cfx[j];
        ay[j] = ay[j] + fr * cfy[j];
      }
    }
    // corrector element force: P+Q+SP+HG are overwritten by the average
#pragma unroll
    for (int j = 0; j < 4; j++) {
      fx[j] = ax[j];
      fy[j] = ay[j];
    }
  } else {
    // ---- corrector force at the half step (zcorrector true)
    force_pq(ph, g.a1, g.a3, g.b1, g.b3, qx, qy, fx, fy);
    if (C.zsp) {
      force_sp(__ldg(C.pmeritreg + ireg), rho, cs2h, xh, yh, F.spmass[iel], fx, fy);
    }
    if (C.zhg) force_hg(__ldg(C.kappareg + ireg), rho, g.vol, S->rdt, u, v, fx, fy);
  }
  F.cnfx[iel] = make_d4(fx[0], fx[1], fx[2], fx[3]);
  F.cnfy[iel] = make_d4(fy[0], fy[1], fy[2], fy[3]);
  F.rho_h[iel] = rho;
  F.cnwt_h[iel] = make_d4(g.w0, g.w1, g.w2, g.w3);
}
#endif

// ================================================================ k_lag_accel

template <int BS, bool BATCH>
__global__ void BL_ACCEL_BOUNDS(BS) k_lag_accel(DevFields F, DevCfg C) {
  const int ind = blockIdx.x * BS + threadIdx.x;
  if (ind >= F.nnd) return;
  const int b = __ldg(F.nc_off + ind), e = __ldg(F.nc_off + ind + 1);
  const DevStep* S = nd_step<BATCH>(F, ind);
  if (halted(S)) return;
  const double dt = S->dt;
  const double zc = C.zerocut;
  // asked for before the gather, used after it
  const int t = __ldg(F.indtype + ind);
  const double u0 = F.ndu[ind], v0 = F.ndv[ind];
  double x = F.ndx[ind], y = F.ndy[ind];
  // hydro_kn_scatteracceleration: corner-major order over ielsort
  double ndm = 0.0, nda = 0.0, fx = 0.0, fy = 0.0;
  for (int k = b; k < e; k++) {
    const int c = __ldg(F.nc_ent + k);
    const int iel = c >> 2, jj = c & 3;
    const double* cm = reinterpret_cast<const double*>(F.cnmass + iel);
    const double cmj = cm[jj];
    const double cw = reinterpret_cast<const double*>(F.cnwt_h + iel)[jj];
    if (gtF(cmj, zc)) {
      ndm = ndm + cmj;
    } else {
      const double cmi = cm[(jj + 3) & 3];
      if (gtF(cmi, zc)) ndm = ndm + cmi;
      else ndm = ndm + F.rho_h[iel] * cw;
    }
    nda = nda + cw;
    fx = fx + reinterpret_cast<const double*>(F.cnfx + iel)[jj];
    fy = fy + reinterpret_cast<const double*>(F.cnfy + iel)[jj];
  }
  // hydro_kn_getacceleration
  const double w1 = C.dencut * nda;
  double ax, ay;
  if (gtF(ndm, w1)) {
    ax = DIV_IN(fx, ndm);
    ay = DIV_IN(fy, ndm);
  } else {
    ax = 0.0;
    ay = 0.0;
  }
  // utils_kn_bc on the accelerations
  if (t == -1) ax = 0.0;
  else if (t == -2) ay = 0.0;
  else if (t == -3) { ax = 0.0; ay = 0.0; }
  const double w2 = ax * ax + ay * ay;
  if (gt_nn(C.accut * C.accut, w2)) {  // w2 is a sum of squares
    ax = 0.0;
    ay = 0.0;
  }
  // hydro_kn_applyacceleration, then both half vertex moves
  const double hdt = 0.5 * dt;
  const double u1 = u0 + dt * ax, v1 = v0 + dt * ay;
  const double ub = u0 + hdt * ax, vb = v0 + hdt * ay;
  x = x + hdt * u0;
  y = y + hdt * v0;
  x = x + hdt * u1;
  y = y + hdt * v1;
  F.ndu[ind] = u1;
  F.ndv[ind] = v1;
  F.ndubar[ind] = ub;
  F.ndvbar[ind] = vb;
  F.ndx[ind] = x;
  F.ndy[ind] = y;
}

// ================================================================ k_lag_state

// ale_active (ale_dr_utils.f90:35-51)
__device__ __forceinline__ bool ale_on(const DevCfg& C, const DevStep* S) {
  if (!C.ale_zexist) return false;
  const double t = S->time;
  return geF(t, C.ale_mintime) && geF(C.ale_maxtime, t);  // the IEEE >= on the integer pipe
}

#if BL_FAST_ALGEBRA
// The volume an element's face sweeps in the remap, from the face vector
// (Dx, Dy) and the differences and sums of the mesh velocity -ubar at its
// ends (a, b): the reference's quarter(a1*b3 - a3*b1) of the quad (x0(a),
// x0(b), x1(b), x1(a)) with x1 = x0 - dt*ubar expands (exactly in real
// arithmetic) to dt/4 * (2 (Dy Su - Dx Sv) + dt (Du Sv - Dv Su)), which also
// avoids the cancellation of subtracting positions at two times.  Run the
// other way (b, a) it is exactly the negative.
__device__ __forceinline__ double swept(double xa, double ya, double ua, double va, double xb,
                                        double yb, double ub, double vb, double dt) {
  const double Dx = xb - xa, Dy = yb - ya, Du = ub - ua, Dv = vb - va;
  const double Su = ub + ua, Sv = vb + va;
  const double A = fma(Dy, Su, -(Dx * Sv)), B = fma(Du, Sv, -(Dv * Su));
  return quarter(dt * fma(dt, B, twice(A)));
}
#endif

// LOOP: in a device loop whose remap follows with the same dt.  What the
// remap then overwrites unread -- the coefficients a1..b3, pressure and sound
// speed -- is left out, and the fast and mixed builds' kernel, which has the
// positions and velocities at hand, leaves the swept volumes of faces 0 and 3
// for k_ale_flux (a step called alone may be followed by anything: it does
// all of its own work, and so does the remap).
template <int BS, bool BATCH, bool LOOP = false>
__global__ void BL_STATE_BOUNDS(BS) k_lag_state(DevFields F, DevCfg C) {
  const int iel = blockIdx.x * BS + threadIdx.x;
  if (iel >= F.nel) return;
  const int4 nd = __ldg(F.ielnd + iel);
  DevStep* S = el_step<BATCH>(F, iel);
  if (halted(S)) return;
  const double dt = S->dt;
  const double zc = C.zerocut;
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  double x[4], y[4], ub[4], vb[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    x[j] = F.ndx[n[j]];
    y[j] = F.ndy[n[j]];
    ub[j] = F.ndubar[n[j]];
    vb[j] = F.ndvbar[n[j]];
  }
  // asked for before the geometry, used after it
  const EosTab mat = eos_tab(C, __ldg(F.ielmat + iel));
  const double m = F.mass[iel], e0 = F.e[iel];
  Iso g = getiso(x, y);
  if (gtF(0.0, g.vol)) note_negvol(F, S, &DevStep::negvol_corr, iel + 1 - el_base<BATCH>(F, iel));
  const double rho = DIV(m, g.vol);
  const d4 f4x = F.cnfx[iel], f4y = F.cnfy[iel];
  const double fx[4] = {f4x.x, f4x.y, f4x.z, f4x.w};
  const double fy[4] = {f4y.x, f4y.y, f4y.z, f4y.w};
  // no work on fluid at rest, with finite forces: then e0 - 0*dt, which is e0
  // bit for bit unless that is a zero itself.  Sedov 512x512 after 60
  // steps: 26.7 -> 23.1 us (exact 42.9 -> 35.0); in motion as before.
  double e = e0;
  const long long still = bits64(ub[0]) | bits64(ub[1]) | bits64(ub[2]) | bits64(ub[3]) |
                          bits64(vb[0]) | bits64(vb[1]) | bits64(vb[2]) | bits64(vb[3]);
  bool rest = (still << 1) == 0 && (bits64(e0) << 1) != 0;
  if (rest) {
    unsigned x = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      x = max(x, (unsigned)(bits64(fx[j]) >> 32) & 0x7ff00000u);
      x = max(x, (unsigned)(bits64(fy[j]) >> 32) & 0x7ff00000u);
    }
    x = max(x, max((unsigned)(bits64(e0) >> 32) & 0x7ff00000u,
                   (unsigned)(bits64(m) >> 32) & 0x7ff00000u));
    rest = x != 0x7ff00000u && gtF(zc, 0.0);
  }
  if (!rest) e = energy_update(e0, m, zc, dt, fx, fy, ub, vb);
  if (!LOOP || !ale_on(C, S)) {
    double p, cs2;
    eos_pc(C, mat, rho, e, p, cs2);
    F.a1[iel] = g.a1;
    F.a2[iel] = g.a2;
    F.a3[iel] = g.a3;
    F.b1[iel] = g.b1;
    F.b2[iel] = g.b2;
    F.b3[iel] = g.b3;
    F.p[iel] = p;
    F.cs2[iel] = cs2;
  } else {
#if BL_FAST_ALGEBRA
    F.fdv0[iel] = swept(x[0], y[0], ub[0], vb[0], x[1], y[1], ub[1], vb[1], dt);
    F.fdv3[iel] = swept(x[3], y[3], ub[3], vb[3], x[0], y[0], ub[0], vb[0], dt);
#endif
  }
  F.cnwt[iel] = make_d4(g.w0, g.w1, g.w2, g.w3);
  const int imx = F.elmx ? F.elmx[iel] : -1;
  // the learned closure (k_mix_closure, beside this kernel) splits a
  // two-material cell's volume change between its materials and updates them
  const bool learned = imx >= 0 && F.closure && F.imxncp[imx] == 2;
  F.vol[iel] = g.vol;
  F.rho[iel] = rho;
  F.e[iel] = e;
  if (imx >= 0 && !learned) {
    const int c0 = F.imxfcp[imx], nc = F.imxncp[imx];
    for (int k = 0; k < nc; k++) {
      const int icp = c0 + k;
      const double fr = F.frvol[icp];
      const d4 a = F.cpfx[icp], b = F.cpfy[icp];
      const double cfx[4] = {a.x, a.y, a.z, a.w}, cfy[4] = {b.x, b.y, b.z, b.w};
      double cu[4], cv[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        cu[j] = fr * ub[j];
        cv[j] = fr * vb[j];
      }
      const double cpm = F.cpm[icp];
      const double cpe = energy_update(F.cpe[icp], cpm, zc, dt, cfx, cfy, cu, cv);
      const double cpv = times4(g.a1 * g.b3 - g.a3 * g.b1) * fr;
      const double cpr = DIV(cpm, cpv);
      double cpp, cpc;
      eos_pc(C, __ldg(F.icpmat + icp), cpr, cpe, cpp, cpc);
      F.cpe[icp] = cpe;
      F.cpvol[icp] = cpv;
      F.cprho[icp] = cpr;
      F.cpp[icp] = cpp;
      F.cpcs2[icp] = cpc;
    }
  }
}

// ================================================================ k_mix_closure

// The learned mixed-cell closure, beside k_lag_state.  For each two-material
// cell the network (tensor cores, 16 cells per warp) predicts the volume
// each material gains over the step beyond the plain closure's share (its
// volume fraction of the cell's change), as a fraction of the cell's volume
// at the start: x_m = norm[20] * y_m.  Its inputs, standardised as
// (f - norm[k]) * norm[10 + k], are the state at the start of the step:
//   0 material 1's volume fraction, 1-2 the densities, 3-4 the pressures,
//   5-6 the sound speeds squared, 7 dV / V^n, 8 dt sqrt(max cs2 / V^n) (a
//   Courant number of the cell), 9 (p1 - p2) / (|p1| + |p2|).
// The exchange used is x = (x_1 - x_2) / 2 into material 1 (x_1 + x_2 = 0
// conserves the cell's volume), limited to the admissible range between 0
// and x_eq, the exchange that equalises the two materials' pressures after
// the plain closure's step (linearised with the bulk moduli rho c^2): the
// closure may relax the materials towards pressure equilibrium, not past it.
// The plain closure is kept in a cell whose outputs are not finite, miss
// conservation (|y_1 + y_2| > norm[21]), lie out of range (farther than
// |x_eq| outside [0, x_eq]) or leave a material a non-positive volume;
// F.mlp_count[1] counts those cells.  Each material's energy takes the plain
// closure's work; with F.closure == 1 the exchanged volume also trades
// energy at the mixture pressure fr_1 p_1 + fr_2 p_2 (the work one material
// does on the other, summing to zero over the cell), with F.closure == 2
// the materials keep their specific energies, so that for ideal gases the
// cell's mixture pressure sum (gamma_m - 1) E_m / V, and with it every later
// element and node field, stays the plain closure's.  Either way the cell's
// volume and total energy, and every element and node field of the step,
// are the plain closure's, and a rejected cell ends exactly as under it.
// In a batch each cell reads the step header of its own mesh.
//
// One dependent chain of loads, network, divides and FP64 on a few warps: 12
// us whatever the number of cells, up to a few thousand.  So it runs beside
// k_lag_state, on a branch of its own (queue_state): the cell's volume at the
// start of the step comes from k_lag_force, the one at its end from the
// vertices, and nothing that one of the two kernels writes is read by the
// other.
constexpr int kClosureWarps = 4;
template <bool BATCH>
__global__ void __launch_bounds__(32 * kClosureWarps) k_mix_closure(DevFields F, DevCfg C) {
  if (!BATCH && halted(F.step)) return;
  extern __shared__ unsigned char smem[];
  mlp::SmemW& w = *reinterpret_cast<mlp::SmemW*>(smem);
  mlp::SmemS* Ss = reinterpret_cast<mlp::SmemS*>(smem + sizeof(mlp::SmemW));
  mlp::copy_weights<32 * kClosureWarps>(w, F.mlp_img);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  mlp::SmemS& s = Ss[warp];
  const int imx = blockIdx.x * (16 * kClosureWarps) + warp * 16 + (lane & 15);
  // lanes l and l + 16 share cell l: the features and the network take one
  // row per cell (lanes 0-15), the FP64 update one material per lane
  const int k = lane >> 4;
  const bool two = imx < F.nmx && F.imxncp[imx] == 2;
  const int iel = two ? F.imxel[imx] : 0;
  const DevStep* S = el_step<BATCH>(F, iel);
  const int4 nd = __ldg(F.ielnd + iel);
  const int n[4] = {nd.x, nd.y, nd.z, nd.w};
  const bool cell = two && !halted(S);
  const double dt = cell ? S->dt : 0.0;
  double V0 = 0.0, V1 = 0.0;
  int c0 = 0;
  if (cell) {
    c0 = F.imxfcp[imx];
    V0 = F.mxv0[imx];
    double x[4], y[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      x[j] = F.ndx[n[j]];
      y[j] = F.ndy[n[j]];
    }
    V1 = getiso(x, y).vol;
  }
  if (lane < 16) {
    float f[mlp::NI];
    if (cell) {
      const double p1 = F.cpp[c0], p2 = F.cpp[c0 + 1];
      const double q1 = F.cpcs2[c0], q2 = F.cpcs2[c0 + 1];
      const double raw[mlp::NI] = {F.frvol[c0], F.cprho[c0], F.cprho[c0 + 1], p1, p2, q1, q2,
                                   (V1 - V0) / V0, dt * sqrt(maxF(q1, q2) / V0),
                                   (p1 - p2) / (absF(p1) + absF(p2) + 1e-300)};
#pragma unroll
      for (int j = 0; j < mlp::NI; j++)
        f[j] = ((float)raw[j] - __ldg(F.mlp_norm + j)) * __ldg(F.mlp_norm + mlp::NI + j);
    }
#pragma unroll
    for (int j = 0; j < 16; j++) s.x[lane][j] = (cell && j < mlp::NI) ? f[j] : 0.0f;
  }
  __syncwarp();
  mlp::forward_warp(w, s);
  // this lane's material: the plain closure's step (k_lag_state's component
  // update), the fallback and the state the admissible range is measured from
  const double zc = C.zerocut;
  const int icp = c0 + k;
  double fr[2] = {0.0, 0.0}, pbar = 0.0;
  double pe = 0.0, pv = 0.0, pr = 0.0, pp = 0.0, pc = 0.0;
  if (cell) {
    fr[0] = F.frvol[c0];
    fr[1] = F.frvol[c0 + 1];
    pbar = fr[0] * F.cpp[c0] + fr[1] * F.cpp[c0 + 1];
    const double frk = k ? fr[1] : fr[0];
    const d4 a = F.cpfx[icp], b = F.cpfy[icp];
    const double cfx[4] = {a.x, a.y, a.z, a.w}, cfy[4] = {b.x, b.y, b.z, b.w};
    double cu[4], cv[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      cu[j] = frk * F.ndubar[n[j]];
      cv[j] = frk * F.ndvbar[n[j]];
    }
    const double cpm = F.cpm[icp];
    pe = energy_update(F.cpe[icp], cpm, zc, dt, cfx, cfy, cu, cv);
    pv = V1 * frk;
    pr = DIV(cpm, pv);
    eos_pc(C, __ldg(F.icpmat + icp), pr, pe, pp, pc);
  }
  // the other material's, from the partner lane
  const double opp = __shfl_xor_sync(0xffffffffu, pp, 16);
  const double opr = __shfl_xor_sync(0xffffffffu, pr, 16);
  const double opc = __shfl_xor_sync(0xffffffffu, pc, 16);
  if (!cell) return;
  const double P0 = k ? opp : pp, P1 = k ? pp : opp;
  const double R0 = k ? opr : pr, R1 = k ? pr : opr;
  const double Q0 = k ? opc : pc, Q1 = k ? pc : opc;
  const double xeq = DIV((P0 - P1) * V1, V0 * (DIV(R0 * Q0, fr[0]) + DIV(R1 * Q1, fr[1])));
  const double lo = fmin(0.0, xeq), hi = fmax(0.0, xeq), m = absF(xeq);
  const float o1 = s.y[lane & 15][0], o2 = s.y[lane & 15][1];
  const double xp = 0.5 * __ldg(F.mlp_norm + 2 * mlp::NI) * ((double)o1 - (double)o2);
  const double xm = fmin(fmax(xp, lo), hi);
  const double xk = k ? -xm : xm;  // this lane's material's share of the exchange
  const bool ok = isfinite(o1) && isfinite(o2) && isfinite(xeq) &&
                  fabsf(o1 + o2) <= __ldg(F.mlp_norm + 2 * mlp::NI + 1) && xp >= lo - m &&
                  xp <= hi + m && V1 * fr[0] + xm * V0 > 0.0 && V1 * fr[1] + (-xm) * V0 > 0.0;
  if (k == 0) {
    atomicAdd(F.mlp_count, 1ull);
    if (!ok) atomicAdd(F.mlp_count + 1, 1ull);
  }
  double cpv = pv, cpe = pe, cpr = pr, cpp = pp, cpc = pc;
  if (ok) {
    const double cpm = F.cpm[icp];
    cpv = pv + xk * V0;
    if (F.closure == 1) cpe = pe - DIV(pbar * (xk * V0), maxF(cpm, zc));
    cpr = DIV(cpm, cpv);
    eos_pc(C, __ldg(F.icpmat + icp), cpr, cpe, cpp, cpc);
    F.frvol[icp] = DIV(cpv, V1);
  }
  F.cpe[icp] = cpe;
  F.cpvol[icp] = cpv;
  F.cprho[icp] = cpr;
  F.cpp[icp] = cpp;
  F.cpcs2[icp] = cpc;
}

// ================================================================ launchers

static constexpr int BS_DT = 128;
static constexpr int BS_EL = 64;   // k_lag_force, k_lag_state
static constexpr int BS_ED = 128;  // k_edge
static constexpr int BS_ND = 128;

// k_getdt blocks of a mesh of nel elements, of all_nel in the context
int getdt_blocks(int nel, int all_nel) {
  const int per = BS_DT * getdt_tiles(all_nel, BS_DT);
  return (nel + per - 1) / per;
}

// a single mesh's grid and number of partials
int getdt_grid(int nel) { return getdt_blocks(nel, nel); }

// k_edge, k_edgevisc: BS - 2 slots or elements a block
static_assert(BS_ED == BS_DT, "one edge_grid");
// the exact build's k_edge: BS / 4 elements a block
[[maybe_unused]] static int face_grid(int nel) { return (nel + BS_ED / 4 - 1) / (BS_ED / 4); }
[[maybe_unused]] static int edge_grid(int n) { return (n + BS_ED - 3) / (BS_ED - 2); }

int getdt_launches(const DevCfg& C) {
#if BL_FAST_ALGEBRA && !BL_MIXED
  (void)C;
  return 2;
#else
  return C.ztq ? 1 : 2;
#endif
}
// (the kernels' POS forms where DevFields::geom_x says so; the exact build
// always takes the positions)
template <bool BATCH>
static void getdt_kernels(const DevFields& F, const DevCfg& C, int grid, cudaStream_t s) {
#if BL_MIXED
  if (!C.ztq) {
    if (F.geom_x) k_edgevisc<BS_DT, BATCH, true><<<edge_grid(F.nel), BS_DT, 0, s>>>(F, C);
    else k_edgevisc<BS_DT, BATCH, false><<<edge_grid(F.nel), BS_DT, 0, s>>>(F, C);
  }
#elif BL_FAST_ALGEBRA
  k_edge<BS_ED, BATCH><<<edge_grid(F.nslot), BS_ED, 0, s>>>(F, C);
#else
  if (!C.ztq) k_edge<BS_ED, BATCH><<<face_grid(F.nel), BS_ED, 0, s>>>(F, C);
#endif
#if BL_FAST_ALGEBRA
  if (F.geom_x) k_getdt<BS_DT, BATCH, true><<<grid, BS_DT, 0, s>>>(F, C);
  else k_getdt<BS_DT, BATCH, false><<<grid, BS_DT, 0, s>>>(F, C);
#else
  k_getdt<BS_DT, BATCH><<<grid, BS_DT, 0, s>>>(F, C);
#endif
}
template <bool BATCH>
static void force_kernel(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  const int g = (F.nel + BS_EL - 1) / BS_EL;
#if BL_FAST_ALGEBRA
  if (F.geom_x) k_lag_force<BS_EL, BATCH, true><<<g, BS_EL, 0, s>>>(F, C);
  else k_lag_force<BS_EL, BATCH, false><<<g, BS_EL, 0, s>>>(F, C);
#else
  k_lag_force<BS_EL, BATCH><<<g, BS_EL, 0, s>>>(F, C);
#endif
}
void launch_getdt(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  getdt_kernels<false>(F, C, getdt_grid(F.nel), s);
}
void launch_lag_force(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  force_kernel<false>(F, C, s);
}
void launch_lag_accel(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  k_lag_accel<BS_ND, false><<<(F.nnd + BS_ND - 1) / BS_ND, BS_ND, 0, s>>>(F, C);
}
void launch_lag_state(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  const int g = (F.nel + BS_EL - 1) / BS_EL;
  if (F.loop_ale) k_lag_state<BS_EL, false, true><<<g, BS_EL, 0, s>>>(F, C);
  else k_lag_state<BS_EL, false><<<g, BS_EL, 0, s>>>(F, C);
}
constexpr size_t kClosureSmem = sizeof(mlp::SmemW) + kClosureWarps * sizeof(mlp::SmemS);
int prepare_mix_closure() {
  return cudaFuncSetAttribute(k_mix_closure<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kClosureSmem) == cudaSuccess &&
                 cudaFuncSetAttribute(k_mix_closure<true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kClosureSmem) == cudaSuccess
             ? 0 : -1;
}
void launch_mix_closure(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  if (!F.closure || F.nmx < 1) return;
  const int per = 16 * kClosureWarps;
  k_mix_closure<false><<<(F.nmx + per - 1) / per, 32 * kClosureWarps, kClosureSmem, s>>>(F, C);
}
void launch_mix_closure_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  if (!F.closure || F.nmx < 1) return;
  const int per = 16 * kClosureWarps;
  k_mix_closure<true><<<(F.nmx + per - 1) / per, 32 * kClosureWarps, kClosureSmem, s>>>(F, C);
}
// a batch of meshes: k_getdt over each mesh's own blocks, the rest over all
// elements or nodes, each reading the step header of its mesh
void launch_getdt_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  getdt_kernels<true>(F, C, F.nblk_batch, s);
}
void launch_lag_force_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  force_kernel<true>(F, C, s);
}
void launch_lag_accel_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  // block size chosen by the batch's autotuner (128, 256 or 512)
  if (F.nd_block == 128) k_lag_accel<128, true><<<(F.nnd + 127) / 128, 128, 0, s>>>(F, C);
  else if (F.nd_block == 512) k_lag_accel<512, true><<<(F.nnd + 511) / 512, 512, 0, s>>>(F, C);
  else k_lag_accel<256, true><<<(F.nnd + 255) / 256, 256, 0, s>>>(F, C);
}
void launch_lag_state_batch(const DevFields& F, const DevCfg& C, cudaStream_t s) {
  const int g = (F.nel + BS_EL - 1) / BS_EL;
  if (F.loop_ale) k_lag_state<BS_EL, true, true><<<g, BS_EL, 0, s>>>(F, C);
  else k_lag_state<BS_EL, true><<<g, BS_EL, 0, s>>>(F, C);
}

}  // namespace BL_NS
}  // namespace bl
