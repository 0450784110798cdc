// step_kernels.cuh -- the time-step kernels: primitive variables,
// compute_rhs (+ txinvr for SP), the BT block-tridiagonal and SP scalar
// pentadiagonal line solves (with ninvr / pinvr / tzetar and add fused into
// their back substitution), and their host-side launchers.
//
// This file is compiled twice, into namespace NPBMZ_NS:
//   exact  with -fmad=false: FP64 in the reference's operation order, no FMA
//          contraction -- bit-for-bit the reference's arithmetic;
//   fast   with -fmad=true : the same FP64 code with FMA contraction, plus the
//          FP32 line-solve (mixed precision) instantiations.
// Every expression keeps the reference's operand order and parenthesisation
// (reference files cited at each kernel).
#pragma once

#include <algorithm>

#include "npbmz_internal.cuh"

#ifndef NPBMZ_NS
#error "NPBMZ_NS must name the variant namespace"
#endif

namespace npbmz {
namespace NPBMZ_NS {

// ============================================================================
// Primitive variables (src/BT/rhs.jl:62-77, src/SP/rhs.jl:62-89), one thread
// per point of the padded plane (padding points compute garbage nobody reads).
// ============================================================================
// xl: x line through the point and its position on it (FP32 BT sweeps of
// the FMA build write the x-line-major state copy there), or xl < 0.
template <bool SP>
__device__ __forceinline__ void prim_point(const Fields& F, const Consts& K, int64_t p, int64_t xl, int xi) {
  const int64_t NP = F.NP;
  {
    const double u1 = F.u[p], u2 = F.u[NP + p], u3 = F.u[2 * NP + p], u4 = F.u[3 * NP + p];
#if NPBMZ_HAS_FP32
    const double rho_inv = nr_rcp(u1);  // within a few ulps of 1/u1 (FMA build)
#else
    const double rho_inv = 1.0e0 / u1;
#endif
    const double square = 0.5e0 * (u2 * u2 + u3 * u3 + u4 * u4) * rho_inv;
    health_check_ek(F, p, u1, F.u[4 * NP + p], square);
    F.prim[PR_RHOI * NP + p] = rho_inv;
    F.prim[PR_US * NP + p] = u2 * rho_inv;
    F.prim[PR_VS * NP + p] = u3 * rho_inv;
    F.prim[PR_WS * NP + p] = u4 * rho_inv;
    F.prim[PR_SQUARE * NP + p] = square;
    F.prim[PR_QS * NP + p] = square * rho_inv;
    if (SP) {
      const double u5 = F.u[4 * NP + p];
      // IEEE square root and divide in both builds: the speed of sound enters
      // the SP adjoint's finite-difference checks, which a few-ulp estimate
      // makes noisy (1/rho above stays on the Newton-Raphson estimate)
      double aux = K.c1c2 * rho_inv * (u5 - square);
      aux = sqrt(aux);
      F.prim[PR_SPEED * NP + p] = aux;
      F.prim[PR_AINV * NP + p] = 1.0e0 / aux;
    }
    if (SP && F.primf) {
      const double v[PS_HI_COUNT] = {rho_inv, u2 * rho_inv, u3 * rho_inv, u4 * rho_inv, F.prim[PR_SPEED * NP + p]};
#pragma unroll
      for (int e = 0; e < PS_HI_COUNT; ++e) {
        float hi, lo;
        split_df(v[e], hi, lo);
        F.primf[e * NP + p] = hi;
        F.primf[(PS_HI_COUNT + e) * NP + p] = lo;
        if (F.pfx && xl >= 0) {
          F.pfx[((int64_t)xi * PS_COUNT + e) * F.nlx + xl] = hi;
          F.pfx[((int64_t)xi * PS_COUNT + PS_HI_COUNT + e) * F.nlx + xl] = lo;
        }
      }
    } else if (F.primf) {
      const double v[PF_HI_COUNT] = {rho_inv, square * rho_inv, u2, u3, u4, F.u[4 * NP + p]};
#pragma unroll
      for (int e = 0; e < PF_HI_COUNT; ++e) {
        float hi, lo;
        split_df(v[e], hi, lo);
        F.primf[e * NP + p] = hi;
        F.primf[(PF_HI_COUNT + e) * NP + p] = lo;
        if (F.pfx && xl >= 0) {
          F.pfx[((int64_t)xi * PF_COUNT + e) * F.nlx + xl] = hi;
          F.pfx[((int64_t)xi * PF_COUNT + PF_HI_COUNT + e) * F.nlx + xl] = lo;
        }
      }
    }
#if NPBMZ_HAS_FP32
    if (F.flux) {
      // point functions of compute_rhs (FMA build): each is differenced by
      // both neighbours, so it is formed once here instead of twice there
      double* X = F.flux;
      const double u5 = F.u[4 * NP + p];
      const double us = u2 * rho_inv, vs = u3 * rho_inv, ws = u4 * rho_inv;
      const double press = K.c2 * (u5 - square);
      const double qs = square * rho_inv, e = u5 * rho_inv;
      // BT: the enthalpy from the pressure (c1 = 1 + c2) and the viscous term
      // without its direction's factor, which compute_rhs applies; class C
      // primitives 380 -> 336 us. SP keeps the expanded forms: with the short
      // ones (529 -> 492 us) its adjoint's central differences, which stand on
      // their rounding noise, went from 6.7e-7 to 3e-6 .. 5e-6 at worst.
      const double h = SP ? K.c1 * u5 - K.c2 * square : u5 + press;
      X[PX_UV * NP + p] = u3 * us;
      X[PX_UW * NP + p] = u4 * us;
      X[PX_VW * NP + p] = u4 * vs;
      X[PX_XX * NP + p] = u2 * us + press;
      X[PX_YY * NP + p] = u3 * vs + press;
      X[PX_ZZ * NP + p] = u4 * ws + press;
      X[PX_EX * NP + p] = h * us;
      X[PX_EY * NP + p] = h * vs;
      X[PX_EZ * NP + p] = h * ws;
      if (SP) {
        X[PX_WX * NP + p] = K.xxcon3 * qs + K.xxcon4 * (us * us) + K.xxcon5 * e;
        X[PX_WY * NP + p] = K.yycon3 * qs + K.yycon4 * (vs * vs) + K.yycon5 * e;
        X[PX_WZ * NP + p] = K.zzcon3 * qs + K.zzcon4 * (ws * ws) + K.zzcon5 * e;
      } else {
        const double base = K.conz1 * qs + K.c1c5 * e;
        X[PX_WX * NP + p] = fma(K.con16 * us, us, base);
        X[PX_WY * NP + p] = fma(K.con16 * vs, vs, base);
        X[PX_WZ * NP + p] = fma(K.con16 * ws, ws, base);
      }
    }
#endif
  }
}

template <bool SP>
__global__ void __launch_bounds__(256) k_prim(Fields F, Consts K, int64_t lo, int64_t hi) {
  for (int64_t p = lo + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < hi; p += (int64_t)gridDim.x * blockDim.x)
    prim_point<SP>(F, K, p, -1, 0);
}

// Over the point work list (zone known): also the x-line-major state copy.
template <bool SP>
// Work-item loop (here and in the other kernels of the batched FMA step):
// CTA b takes items b, b + gridDim.x, ...; launched with one CTA per item, or
// as a persistent kernel with as many CTAs as fit on the SMs (NPBMZ_PERSIST).
__global__ void __launch_bounds__(128) k_prim_w(Fields F, Consts K, const Work* __restrict__ work, int nwork) {
  for (int it = blockIdx.x; it < nwork; it += gridDim.x) {
    const Work w = work[it];
    const ZoneDev Z = F.zones[w.zone];
    const int q = w.first + threadIdx.x;
    if (q >= Z.nx * Z.ny * Z.nz) continue;
    const int i = q % Z.nx, j = (q / Z.nx) % Z.ny, k = q / (Z.nx * Z.ny);
    prim_point<SP>(F, K, Z.off + q, xline_of(Z, j, k), i);
  }
}

// ============================================================================
// compute_rhs (src/BT/rhs.jl:4-460; SP src/SP/rhs.jl:3-452 -- the flux and
// dissipation statements are identical) and, when TX (the SP step), txinvr
// (src/SP/txinvr.jl:5-56).  One thread per zone point; boundary points copy
// the forcing, as the reference's `rhs = forcing` over the whole cell does.
// Per element the order of updates is the reference's: forcing, xi flux, xi
// dissipation, eta flux, eta dissipation, zeta flux, zeta dissipation, *dt.
// NORM: also accumulate this CTA's sum of rhs^2 (interior, before txinvr)
// into partials[blockIdx.x][5] (each CTA covers points of one zone).
// ============================================================================

// Fourth-order dissipation term at position q of an axis of n points
// (1 <= q <= n-2).  On six points and more one of the reference's start,
// middle and end stencils applies: the middle one, whose missing terms enter
// as zeros (0 + x and x - 0 are x), with 5 instead of 6 at the centre of the
// outermost two -- no lane diverges, and the products with 4 and with dssp
// (0.25 for every problem: set_constants) are exact, so fma rounds them and
// their sum once, as the separate operations do.
constexpr double DSSP = 0.25;
__device__ __forceinline__ double dissip(double r, int q, int n, double um2, double um1, double u0, double up1,
                                         double up2) {
  if (n >= 6) {
    const double a = q >= 3 ? um2 : 0.0, b = q >= 2 ? um1 : 0.0, d = q <= n - 3 ? up1 : 0.0, e = q <= n - 4 ? up2 : 0.0;
    const double w = q == 1 || q == n - 2 ? 5.0e0 : 6.0e0;
    return fma(-DSSP, fma(-4.0e0, d, fma(-4.0e0, b, a) + w * u0) + e, r);
  }
  // shorter axes: several stencils at one point, in the reference's order
  if (q == 1) r -= DSSP * (5.0e0 * u0 - 4.0e0 * up1 + up2);
  if (q == 2) r -= DSSP * (-4.0e0 * um1 + 6.0e0 * u0 - 4.0e0 * up1 + up2);
  if (q >= 3 && q <= n - 4) r -= DSSP * (um2 - 4.0e0 * um1 + 6.0 * u0 - 4.0e0 * up1 + up2);
  if (q == n - 3) r -= DSSP * (um2 - 4.0e0 * um1 + 6.0e0 * u0 - 4.0e0 * up1);
  if (q == n - 2) r -= DSSP * (um2 - 4.0e0 * um1 + 5.0e0 * u0);
  return r;
}

// Safe neighbour load along an axis: positions outside 0..n-1 are never used
// by dissip() (their stencil weight is absent), so they read the centre.
__device__ __forceinline__ double ld_axis(const double* __restrict__ a, int64_t p, int64_t st, int q, int d, int n) {
  const int qq = q + d;
  return (qq >= 0 && qq < n) ? a[p + d * st] : a[p];
}

// up - 2 u0 + um, left to right: 2 u0 is exact, so fma rounds the difference once
__device__ __forceinline__ double d2(double up, double u0, double um) { return fma(-2.0e0, u0, up) + um; }

// Bound by the FP64 pipe in both builds; this kernel is the exact build's:
// 304x208x17 938 -> 560 us with the products with 2, 4 and dssp fused (exactly)
// into the sums and no branch per stencil.
// One thread per INTERIOR point of a zone (the work list counts interior
// points only): the boundary rhs equals the forcing and no solve rewrites
// it, so it is set when the forcing or rhs is set, not every step.
template <bool TX, bool NORM>
__global__ void __launch_bounds__(128) k_rhs(Fields F, Consts K, const Work* __restrict__ work,
                                             double* __restrict__ partials) {
  __shared__ double red[5 * 128];
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int64_t NP = F.NP;
  const int ix = Z.nx - 2, iy = Z.ny - 2;
  const int ni = ix * iy * (Z.nz - 2);
  const int t = w.first + threadIdx.x;
  double sq[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (t < ni) {
    const int i = 1 + t % ix, j = 1 + (t / ix) % iy, k = 1 + t / (ix * iy);
    const int64_t p = Z.off + ((int64_t)k * Z.ny + j) * Z.nx + i;
    {
      const double* __restrict__ u = F.u;
      const double* __restrict__ pr = F.prim;
      const double* us = pr + PR_US * NP;
      const double* vs = pr + PR_VS * NP;
      const double* ws = pr + PR_WS * NP;
      const double* qs = pr + PR_QS * NP;
      const double* sqr = pr + PR_SQUARE * NP;
      const double* ri = pr + PR_RHOI * NP;
      double r[5];
      for (int m = 0; m < 5; ++m) r[m] = F.forcing[m * NP + p];
      const int64_t sx = 1, sy = Z.nx, sz = (int64_t)Z.nx * Z.ny;
      const double c1 = K.c1, c2 = K.c2, con43 = K.con43;
      // ---------------- xi direction ----------------
      {
        const int64_t a = p + sx, b = p - sx;
        const double uijk = us[p], up1 = us[a], um1 = us[b];
        r[0] += K.dx1tx1 * d2(u[a], u[p], u[b]) - K.tx2 * (u[NP + a] - u[NP + b]);
        r[1] += K.dx2tx1 * d2(u[NP + a], u[NP + p], u[NP + b]) + K.xxcon2 * con43 * d2(up1, uijk, um1) -
                K.tx2 * (u[NP + a] * up1 - u[NP + b] * um1 + (u[4 * NP + a] - sqr[a] - u[4 * NP + b] + sqr[b]) * c2);
        r[2] += K.dx3tx1 * d2(u[2 * NP + a], u[2 * NP + p], u[2 * NP + b]) +
                K.xxcon2 * d2(vs[a], vs[p], vs[b]) - K.tx2 * (u[2 * NP + a] * up1 - u[2 * NP + b] * um1);
        r[3] += K.dx4tx1 * d2(u[3 * NP + a], u[3 * NP + p], u[3 * NP + b]) +
                K.xxcon2 * d2(ws[a], ws[p], ws[b]) - K.tx2 * (u[3 * NP + a] * up1 - u[3 * NP + b] * um1);
        r[4] += K.dx5tx1 * d2(u[4 * NP + a], u[4 * NP + p], u[4 * NP + b]) +
                K.xxcon3 * d2(qs[a], qs[p], qs[b]) + K.xxcon4 * d2(up1 * up1, uijk * uijk, um1 * um1) +
                K.xxcon5 * d2(u[4 * NP + a] * ri[a], u[4 * NP + p] * ri[p], u[4 * NP + b] * ri[b]) -
                K.tx2 * ((c1 * u[4 * NP + a] - c2 * sqr[a]) * up1 - (c1 * u[4 * NP + b] - c2 * sqr[b]) * um1);
        for (int m = 0; m < 5; ++m) {
          const double* um = u + m * NP;
          r[m] = dissip(r[m], i, Z.nx, ld_axis(um, p, sx, i, -2, Z.nx), um[p - sx], um[p], um[p + sx],
                       ld_axis(um, p, sx, i, 2, Z.nx));
        }
      }
      // ---------------- eta direction ----------------
      {
        const int64_t a = p + sy, b = p - sy;
        const double vijk = vs[p], vp1 = vs[a], vm1 = vs[b];
        r[0] += K.dy1ty1 * d2(u[a], u[p], u[b]) - K.ty2 * (u[2 * NP + a] - u[2 * NP + b]);
        r[1] += K.dy2ty1 * d2(u[NP + a], u[NP + p], u[NP + b]) + K.yycon2 * d2(us[a], us[p], us[b]) -
                K.ty2 * (u[NP + a] * vp1 - u[NP + b] * vm1);
        r[2] += K.dy3ty1 * d2(u[2 * NP + a], u[2 * NP + p], u[2 * NP + b]) +
                K.yycon2 * con43 * d2(vp1, vijk, vm1) -
                K.ty2 * (u[2 * NP + a] * vp1 - u[2 * NP + b] * vm1 + (u[4 * NP + a] - sqr[a] - u[4 * NP + b] + sqr[b]) * c2);
        r[3] += K.dy4ty1 * d2(u[3 * NP + a], u[3 * NP + p], u[3 * NP + b]) +
                K.yycon2 * d2(ws[a], ws[p], ws[b]) - K.ty2 * (u[3 * NP + a] * vp1 - u[3 * NP + b] * vm1);
        r[4] += K.dy5ty1 * d2(u[4 * NP + a], u[4 * NP + p], u[4 * NP + b]) +
                K.yycon3 * d2(qs[a], qs[p], qs[b]) + K.yycon4 * d2(vp1 * vp1, vijk * vijk, vm1 * vm1) +
                K.yycon5 * d2(u[4 * NP + a] * ri[a], u[4 * NP + p] * ri[p], u[4 * NP + b] * ri[b]) -
                K.ty2 * ((c1 * u[4 * NP + a] - c2 * sqr[a]) * vp1 - (c1 * u[4 * NP + b] - c2 * sqr[b]) * vm1);
        for (int m = 0; m < 5; ++m) {
          const double* um = u + m * NP;
          r[m] = dissip(r[m], j, Z.ny, ld_axis(um, p, sy, j, -2, Z.ny), um[p - sy], um[p], um[p + sy],
                       ld_axis(um, p, sy, j, 2, Z.ny));
        }
      }
      // ---------------- zeta direction ----------------
      {
        const int64_t a = p + sz, b = p - sz;
        const double wijk = ws[p], wp1 = ws[a], wm1 = ws[b];
        r[0] += K.dz1tz1 * d2(u[a], u[p], u[b]) - K.tz2 * (u[3 * NP + a] - u[3 * NP + b]);
        r[1] += K.dz2tz1 * d2(u[NP + a], u[NP + p], u[NP + b]) + K.zzcon2 * d2(us[a], us[p], us[b]) -
                K.tz2 * (u[NP + a] * wp1 - u[NP + b] * wm1);
        r[2] += K.dz3tz1 * d2(u[2 * NP + a], u[2 * NP + p], u[2 * NP + b]) +
                K.zzcon2 * d2(vs[a], vs[p], vs[b]) - K.tz2 * (u[2 * NP + a] * wp1 - u[2 * NP + b] * wm1);
        r[3] += K.dz4tz1 * d2(u[3 * NP + a], u[3 * NP + p], u[3 * NP + b]) +
                K.zzcon2 * con43 * d2(wp1, wijk, wm1) -
                K.tz2 * (u[3 * NP + a] * wp1 - u[3 * NP + b] * wm1 + (u[4 * NP + a] - sqr[a] - u[4 * NP + b] + sqr[b]) * c2);
        r[4] += K.dz5tz1 * d2(u[4 * NP + a], u[4 * NP + p], u[4 * NP + b]) +
                K.zzcon3 * d2(qs[a], qs[p], qs[b]) + K.zzcon4 * d2(wp1 * wp1, wijk * wijk, wm1 * wm1) +
                K.zzcon5 * d2(u[4 * NP + a] * ri[a], u[4 * NP + p] * ri[p], u[4 * NP + b] * ri[b]) -
                K.tz2 * ((c1 * u[4 * NP + a] - c2 * sqr[a]) * wp1 - (c1 * u[4 * NP + b] - c2 * sqr[b]) * wm1);
        for (int m = 0; m < 5; ++m) {
          const double* um = u + m * NP;
          r[m] = dissip(r[m], k, Z.nz, ld_axis(um, p, sz, k, -2, Z.nz), um[p - sz], um[p], um[p + sz],
                       ld_axis(um, p, sz, k, 2, Z.nz));
        }
      }
      for (int m = 0; m < 5; ++m) r[m] *= K.dt;
      if (NORM)
        for (int m = 0; m < 5; ++m) sq[m] = r[m] * r[m];
      if (TX) {
        // txinvr (src/SP/txinvr.jl:28-49)
        const double ru1 = ri[p], uu = us[p], vv = vs[p], ww = ws[p], ac = pr[PR_SPEED * NP + p];
        const double ac2inv = 1.0 / (ac * ac);
        const double r1 = r[0], r2 = r[1], r3 = r[2], r4 = r[3], r5 = r[4];
        const double t1 = K.c2 * ac2inv * (qs[p] * r1 - uu * r2 - vv * r3 - ww * r4 + r5);
        const double t2 = K.bt * ru1 * (uu * r1 - r2);
        const double t3 = (K.bt * ru1 * ac) * t1;
        r[0] = r1 - t1;
        r[1] = -ru1 * (ww * r1 - r4);
        r[2] = ru1 * (vv * r1 - r3);
        r[3] = -t2 + t3;
        r[4] = t2 + t3;
      }
      for (int m = 0; m < 5; ++m) F.rhs[m * NP + p] = r[m];
    }
  }
  if (NORM) {
    block_sum5(sq, red);
    if (threadIdx.x == 0)
      for (int m = 0; m < 5; ++m) partials[blockIdx.x * 5 + m] = sq[m];
  }
}

#if NPBMZ_HAS_FP32
// ============================================================================
// compute_rhs, FMA build: the same terms as k_rhs, regrouped to cut FP64
// work (this path is bound by GB300's FP64 pipe, not by HBM):
//   - the fluxes and viscous energy terms come from the point functions the
//     primitive kernel wrote (PX_*), each formed once per point;
//   - per direction and variable, the second difference d*t1*D2(u) and the
//     dissipation are one 5-point stencil with weights from LinWeights,
//     staged in shared memory;
//   - the momentum viscous terms difference the velocity planes.
// The sum is algebraically the reference's; rounding differs (within 1e-12
// of the oracle, tested).
// ============================================================================
__device__ __forceinline__ int dissip_class(int q, int n) {
  return (q == 1) | ((q == 2) << 1) | ((q >= 3 && q <= n - 4) << 2) | ((q == n - 3) << 3) | ((q == n - 2) << 4);
}

// One direction: stride st, position q of n, weights W (5; the centre one,
// W[2], is summed over the directions by the caller), flux planes of
// variables 1..4 (fx[0..3]), normal momentum plane (variable a = 1 + dir),
// velocity-term factors vc[3] (their centre term likewise), viscous energy
// plane wv and its factor kw, t2; every factor carries dt.
__device__ __forceinline__ void rhs_dir(double r[5], const double* __restrict__ u, int64_t NP, int64_t p, int64_t st,
                                        int q, int n, const double* __restrict__ W, const double* const fx[4],
                                        const double* __restrict__ un, const double* const vel[3], const double vc[3],
                                        const double* __restrict__ wv, double t2, double kw) {
  const int64_t pm2 = q >= 2 ? p - 2 * st : p;
  const int64_t pp2 = q + 2 <= n - 1 ? p + 2 * st : p;
  const double w0 = W[0], w1 = W[1], w3 = W[3], w4 = W[4];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const double* um = u + m * NP;
    double s = fma(w1, um[p - st], r[m]);
    s = fma(w3, um[p + st], s);
    s = fma(w0, um[pm2], s);
    r[m] = fma(w4, um[pp2], s);
  }
  r[0] = fma(-t2, un[p + st] - un[p - st], r[0]);
#pragma unroll
  for (int m = 0; m < 4; ++m) r[m + 1] = fma(-t2, fx[m][p + st] - fx[m][p - st], r[m + 1]);
#pragma unroll
  for (int m = 0; m < 3; ++m) r[m + 1] = fma(vc[m], vel[m][p + st] + vel[m][p - st], r[m + 1]);
  r[4] = fma(kw, (wv[p + st] + wv[p - st]) - 2.0 * wv[p], r[4]);
}

// One work item (128 interior points of one zone) of compute_rhs; wt: the
// dissipation weights in shared memory, red: the NORM reduction scratch.
template <bool TX, bool NORM>
__device__ __forceinline__ void rhs_flux_item(const Fields& F, const Consts& K, const RhsF64Consts& RC, const Work w,
                                              int it, double* __restrict__ partials, const double* wt, double* red) {
  const ZoneDev Z = F.zones[w.zone];
  const int64_t NP = F.NP;
  const int ix = Z.nx - 2, iy = Z.ny - 2;
  const int ni = ix * iy * (Z.nz - 2);
  const int t = w.first + threadIdx.x;
  double sq[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (t < ni) {
    const int i = 1 + t % ix, j = 1 + (t / ix) % iy, k = 1 + t / (ix * iy);
    const int64_t p = Z.off + ((int64_t)k * Z.ny + j) * Z.nx + i;
    const double* __restrict__ u = F.u;
    const double* __restrict__ pr = F.prim;
    const double* __restrict__ X = F.flux;
    const double* vel[3] = {pr + PR_US * NP, pr + PR_VS * NP, pr + PR_WS * NP};
    double r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = F.fdt[m * NP + p];
    const double* Wx = wt + (0 * 32 + dissip_class(i, Z.nx)) * 5;
    const double* Wy = wt + (1 * 32 + dissip_class(j, Z.ny)) * 5;
    const double* Wz = wt + (2 * 32 + dissip_class(k, Z.nz)) * 5;
    {
      const double* fx[4] = {X + PX_XX * NP, X + PX_UV * NP, X + PX_UW * NP, X + PX_EX * NP};
      rhs_dir(r, u, NP, p, 1, i, Z.nx, Wx, fx, u + NP, vel, RC.vc[0], X + PX_WX * NP, RC.t2[0], RC.kw[0]);
    }
    {
      const double* fx[4] = {X + PX_UV * NP, X + PX_YY * NP, X + PX_VW * NP, X + PX_EY * NP};
      rhs_dir(r, u, NP, p, Z.nx, j, Z.ny, Wy, fx, u + 2 * NP, vel, RC.vc[1], X + PX_WY * NP, RC.t2[1], RC.kw[1]);
    }
    {
      const double* fx[4] = {X + PX_UW * NP, X + PX_VW * NP, X + PX_ZZ * NP, X + PX_EZ * NP};
      rhs_dir(r, u, NP, p, (int64_t)Z.nx * Z.ny, k, Z.nz, Wz, fx, u + 3 * NP, vel, RC.vc[2], X + PX_WZ * NP,
              RC.t2[2], RC.kw[2]);
    }
    // centre point: the three directions' stencil weights and velocity
    // factors summed first
    const double wc = (Wx[2] + Wy[2]) + Wz[2];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = fma(wc, u[m * NP + p], r[m]);
#pragma unroll
    for (int m = 0; m < 3; ++m) r[m + 1] = fma(RC.vcc[m], vel[m][p], r[m + 1]);
    if (NORM)
#pragma unroll
      for (int m = 0; m < 5; ++m) sq[m] = r[m] * r[m];
    if (TX) {
      // txinvr (src/SP/txinvr.jl:28-49); 1/speed^2 as ainv^2
      const double ru1 = pr[PR_RHOI * NP + p], uu = vel[0][p], vv = vel[1][p], ww = vel[2][p];
      const double ac = pr[PR_SPEED * NP + p], ainv = pr[PR_AINV * NP + p];
      const double ac2inv = ainv * ainv;
      const double r1 = r[0], r2 = r[1], r3 = r[2], r4 = r[3], r5 = r[4];
      const double t1 = K.c2 * ac2inv * (pr[PR_QS * NP + p] * r1 - uu * r2 - vv * r3 - ww * r4 + r5);
      const double t2 = K.bt * ru1 * (uu * r1 - r2);
      const double t3 = (K.bt * ru1 * ac) * t1;
      r[0] = r1 - t1;
      r[1] = -ru1 * (ww * r1 - r4);
      r[2] = ru1 * (vv * r1 - r3);
      r[3] = -t2 + t3;
      r[4] = t2 + t3;
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) F.rhs[m * NP + p] = r[m];
    if (F.rdx) {  // b of the x sweep, x-line-major
      const int64_t xl = xline_of(Z, j, k);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float hi, lo;
        split_df(r[m], hi, lo);
        F.rdx[((int64_t)i * 10 + m) * F.nlx + xl] = hi;
        F.rdx[((int64_t)i * 10 + 5 + m) * F.nlx + xl] = lo;
      }
    } else if (F.rdf) {
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float hi, lo;
        split_df(r[m], hi, lo);
        F.rdf[m * NP + p] = hi;
        F.rdf[(5 + m) * NP + p] = lo;
      }
    }
  }
  if (NORM) {
    block_sum5(sq, red);
    if (threadIdx.x == 0)
      for (int m = 0; m < 5; ++m) partials[it * 5 + m] = sq[m];
  }
}

template <bool TX, bool NORM>
__global__ void __launch_bounds__(128) k_rhs_flux(Fields F, Consts K, RhsF64Consts RC, const Work* __restrict__ work,
                                                  int nwork, double* __restrict__ partials) {
  __shared__ double red[NORM ? 5 * 128 : 1];
  __shared__ double wt[3 * 32 * 5];
  for (int e = threadIdx.x; e < 3 * 32 * 5; e += blockDim.x) wt[e] = (&RC.w[0][0][0])[e];
  __syncthreads();
  for (int it = blockIdx.x; it < nwork; it += gridDim.x) rhs_flux_item<TX, NORM>(F, K, RC, work[it], it, partials, wt, red);
}

// The two end points of every x line in the x-line-major double-float rhs
// copy: the forcing, as rhs holds there (one thread per x line).
__global__ void __launch_bounds__(128) k_xline_ends(Fields F, const Work* __restrict__ work) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, 0)) return;
  int64_t base, st;
  line_geometry(Z, 0, line, base, st);
  const int64_t gl = Z.lineoff[0] + line;
  const int ends[2] = {0, Z.nx - 1};
#pragma unroll
  for (int e = 0; e < 2; ++e)
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double v = F.forcing[m * F.NP + base + ends[e]];
      const float hi = __double2float_rn(v);
      F.rdx[((int64_t)ends[e] * 10 + m) * F.nlx + gl] = hi;
      F.rdx[((int64_t)ends[e] * 10 + 5 + m) * F.nlx + gl] = __double2float_rn(v - (double)hi);
    }
}

// dst = a * src (n values)
__global__ void __launch_bounds__(256) k_scale(const double* __restrict__ src, double* __restrict__ dst, double a,
                                               int64_t n) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    dst[t] = a * src[t];
}

// dst (double-float planes 0..4 hi, 5..9 lo) <- src (5 FP64 planes)
__global__ void __launch_bounds__(256) k_split_df(const double* __restrict__ src, float* __restrict__ dst, int64_t NP) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 5 * NP; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t / NP, p = t - m * NP;
    const double v = src[t];
    const float hi = __double2float_rn(v);
    dst[m * NP + p] = hi;
    dst[(5 + m) * NP + p] = __double2float_rn(v - (double)hi);
  }
}
#endif  // NPBMZ_HAS_FP32

// ============================================================================
// BT block-tridiagonal line solve, one thread per line.
// Reference: x_solve_cell / y_solve_cell / z_solve_cell and the back
// substitutions (src/BT/x_solve.jl:444-488,501-1746, src/BT/y_solve.jl:443-820,
// src/BT/z_solve.jl:438-864) with matvec_sub, matmul_sub2, binvcrhs, binvrhs
// (src/BT/solve_subs.jl:4-37,333-460,468-862).
//
// The Jacobians fjac/njac have structural zeros; terms with a structural
// zero factor are skipped.  That is exact: in the reference such a term
// contributes +-0, and x - (+-0) == x for every nonzero x.  The boundary
// steps (binvcrhs at point 0 with B = I, C = 0; binvrhs at point n-1 with
// A = 0, B = I; back substitution at point 0 with C = 0) are exact no-ops in
// the reference and are skipped for the same reason.
// C'_p (the 5x5 block left by binvcrhs) goes to the line scratch
// lhsc[(p*25 + e) * nlt + global_line] (coalesced across the CTA's lines);
// the forward-eliminated rhs goes back into rhs in place.
// ============================================================================

// Structural nonzeros of fjac / njac per sweep direction.
template <int DIR>
__host__ __device__ constexpr bool fnz(int a, int b) {
  return DIR == 0 ? (a == 0 ? b == 1 : a == 1 ? true : a == 2 ? (b <= 2) : a == 3 ? (b == 0 || b == 1 || b == 3) : true)
       : DIR == 1 ? (a == 0 ? b == 2 : a == 1 ? (b <= 2) : a == 2 ? true : a == 3 ? (b == 0 || b == 2 || b == 3) : true)
                  : (a == 0 ? b == 3 : a == 1 ? (b == 0 || b == 1 || b == 3) : a == 2 ? (b == 0 || b == 2 || b == 3) : true);
}
__host__ __device__ constexpr bool nnz(int a, int b) {
  return a == 0 ? false : a == 4 ? true : (b == 0 || b == a);
}
template <int DIR>
__host__ __device__ constexpr bool anz(int a, int b) { return fnz<DIR>(a, b) || nnz(a, b) || a == b; }

#if !NPBMZ_HAS_FP32  // the exact build's elimination; the FMA build's: bt_lines.cuh
__host__ __device__ constexpr bool bnz(int a, int b) { return nnz(a, b) || a == b; }

// fjac / njac at one point (src/BT/x_solve.jl:536-609, y_solve.jl:543-613,
// z_solve.jl:537-618); only structural nonzeros are written.
template <int DIR>
__device__ __forceinline__ void bt_jac(const Consts& K, double tmp1, double u2, double u3, double u4, double u5,
                                       double q, double f[5][5], double n[5][5]) {
  const double c1 = K.c1, c2 = K.c2, c3c4 = K.c3c4;
  const double c1345 = K.c1345, con43 = K.con43;
  const double tmp2 = tmp1 * tmp1;
  const double tmp3 = tmp1 * tmp2;
  if (DIR == 0) {
    f[0][1] = 1.0;
    f[1][0] = -(u2 * tmp2 * u2) + c2 * q;
    f[1][1] = (2.0 - c2) * (u2 * tmp1);
    f[1][2] = -c2 * (u3 * tmp1);
    f[1][3] = -c2 * (u4 * tmp1);
    f[1][4] = c2;
    f[2][0] = -(u2 * u3) * tmp2;
    f[2][1] = u3 * tmp1;
    f[2][2] = u2 * tmp1;
    f[3][0] = -(u2 * u4) * tmp2;
    f[3][1] = u4 * tmp1;
    f[3][3] = u2 * tmp1;
    f[4][0] = (c2 * 2.0 * q - c1 * (u5 * tmp1)) * (u2 * tmp1);
    f[4][1] = c1 * u5 * tmp1 - c2 * (u2 * u2 * tmp2 + q);
    f[4][2] = -c2 * (u3 * u2) * tmp2;
    f[4][3] = -c2 * (u4 * u2) * tmp2;
    f[4][4] = c1 * (u2 * tmp1);
    n[1][0] = -con43 * c3c4 * tmp2 * u2;
    n[1][1] = con43 * c3c4 * tmp1;
    n[2][0] = -c3c4 * tmp2 * u3;
    n[2][2] = c3c4 * tmp1;
    n[3][0] = -c3c4 * tmp2 * u4;
    n[3][3] = c3c4 * tmp1;
    n[4][0] = -(con43 * c3c4 - c1345) * tmp3 * (u2 * u2) - (c3c4 - c1345) * tmp3 * (u3 * u3) -
              (c3c4 - c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5;
    n[4][1] = (con43 * c3c4 - c1345) * tmp2 * u2;
    n[4][2] = (c3c4 - c1345) * tmp2 * u3;
    n[4][3] = (c3c4 - c1345) * tmp2 * u4;
    n[4][4] = (c1345) * tmp1;
  } else if (DIR == 1) {
    f[0][2] = 1.0;
    f[1][0] = -(u2 * u3) * tmp2;
    f[1][1] = u3 * tmp1;
    f[1][2] = u2 * tmp1;
    f[2][0] = -(u3 * u3 * tmp2) + c2 * q;
    f[2][1] = -c2 * u2 * tmp1;
    f[2][2] = (2.0 - c2) * u3 * tmp1;
    f[2][3] = -c2 * u4 * tmp1;
    f[2][4] = c2;
    f[3][0] = -(u3 * u4) * tmp2;
    f[3][2] = u4 * tmp1;
    f[3][3] = u3 * tmp1;
    f[4][0] = (c2 * 2.0 * q - c1 * u5 * tmp1) * u3 * tmp1;
    f[4][1] = -c2 * u2 * u3 * tmp2;
    f[4][2] = c1 * u5 * tmp1 - c2 * (q + u3 * u3 * tmp2);
    f[4][3] = -c2 * (u3 * u4) * tmp2;
    f[4][4] = c1 * u3 * tmp1;
    n[1][0] = -c3c4 * tmp2 * u2;
    n[1][1] = c3c4 * tmp1;
    n[2][0] = -con43 * c3c4 * tmp2 * u3;
    n[2][2] = con43 * c3c4 * tmp1;
    n[3][0] = -c3c4 * tmp2 * u4;
    n[3][3] = c3c4 * tmp1;
    n[4][0] = -(c3c4 - c1345) * tmp3 * (u2 * u2) - (con43 * c3c4 - c1345) * tmp3 * (u3 * u3) -
              (c3c4 - c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5;
    n[4][1] = (c3c4 - c1345) * tmp2 * u2;
    n[4][2] = (con43 * c3c4 - c1345) * tmp2 * u3;
    n[4][3] = (c3c4 - c1345) * tmp2 * u4;
    n[4][4] = (c1345) * tmp1;
  } else {
    const double c3 = K.c3, c4 = K.c4;
    f[0][3] = 1.0;
    f[1][0] = -(u2 * u4) * tmp2;
    f[1][1] = u4 * tmp1;
    f[1][3] = u2 * tmp1;
    f[2][0] = -(u3 * u4) * tmp2;
    f[2][2] = u4 * tmp1;
    f[2][3] = u3 * tmp1;
    f[3][0] = -(u4 * u4 * tmp2) + c2 * q;
    f[3][1] = -c2 * u2 * tmp1;
    f[3][2] = -c2 * u3 * tmp1;
    f[3][3] = (2.0 - c2) * u4 * tmp1;
    f[3][4] = c2;
    f[4][0] = (c2 * 2.0 * q - c1 * (u5 * tmp1)) * (u4 * tmp1);
    f[4][1] = -c2 * (u2 * u4) * tmp2;
    f[4][2] = -c2 * (u3 * u4) * tmp2;
    f[4][3] = c1 * (u5 * tmp1) - c2 * (q + u4 * u4 * tmp2);
    f[4][4] = c1 * u4 * tmp1;
    n[1][0] = -c3c4 * tmp2 * u2;
    n[1][1] = c3c4 * tmp1;
    n[2][0] = -c3c4 * tmp2 * u3;
    n[2][2] = c3c4 * tmp1;
    n[3][0] = -con43 * c3c4 * tmp2 * u4;
    n[3][3] = con43 * c3 * c4 * tmp1;
    n[4][0] = -(c3c4 - c1345) * tmp3 * (u2 * u2) - (c3c4 - c1345) * tmp3 * (u3 * u3) -
              (con43 * c3c4 - c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5;
    n[4][1] = (c3c4 - c1345) * tmp2 * u2;
    n[4][2] = (c3c4 - c1345) * tmp2 * u3;
    n[4][3] = (con43 * c3c4 - c1345) * tmp2 * u4;
    n[4][4] = (c1345) * tmp1;
  }
}

// f <- tmp2 * f, n <- tmp1 * n: the products lhsa, lhsb and lhsc are sums of
// (-tmp2 * f is their negative, tmp1 * 2.0 * n their double, both exactly).
template <int DIR>
__device__ __forceinline__ void bt_scale(double f[5][5], double n[5][5], double tmp1, double tmp2) {
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      if (fnz<DIR>(a, b)) f[a][b] = tmp2 * f[a][b];
      if (nnz(a, b)) n[a][b] = tmp1 * n[a][b];
    }
}

// lhsa at the point after the Jacobian point: -tmp2*f - tmp1*n - tmp1*d (diag).
template <int DIR>
__device__ __forceinline__ void bt_asm_a(const double f[5][5], const double n[5][5], double tmp1, const double dd[5],
                                         double A[5][5]) {
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      if (!anz<DIR>(a, b)) continue;
      double t;
      bool have = false;
      if (fnz<DIR>(a, b)) { t = -f[a][b]; have = true; }
      if (nnz(a, b)) { t = have ? t - n[a][b] : -n[a][b]; have = true; }
      if (a == b) { t = have ? t - tmp1 * dd[a] : -(tmp1 * dd[a]); }
      A[a][b] = t;
    }
}

// lhsc at the point before the Jacobian point: tmp2*f - tmp1*n - tmp1*d (diag).
template <int DIR>
__device__ __forceinline__ void bt_asm_c(const double f[5][5], const double n[5][5], double tmp1, const double dd[5],
                                         double C[5][5]) {
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      double t = 0.0;
      bool have = false;
      if (fnz<DIR>(a, b)) { t = f[a][b]; have = true; }
      if (nnz(a, b)) { t = have ? t - n[a][b] : -n[a][b]; have = true; }
      if (a == b) { t = have ? t - tmp1 * dd[a] : -(tmp1 * dd[a]); }
      C[a][b] = t;
    }
}

// lhsb at the Jacobian point: 1 + tmp1*2*n + tmp1*2*d (diag), tmp1*2*n off-diag.
__device__ __forceinline__ void bt_asm_b(const double n[5][5], double tmp1, const double dd[5], double B[5][5]) {
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      if (!bnz(a, b)) continue;
      if (a == b) {
        double t = 1.0;
        if (nnz(a, b)) t = fma(2.0, n[a][b], t);
        B[a][b] = t + tmp1 * 2.0 * dd[a];
      } else {
        B[a][b] = 2.0 * n[a][b];
      }
    }
}
#endif

// Pivot reciprocal: in FP64 the reference's division, in the FMA build within
// one ulp; in the FP32 solves, which a double-float refinement corrects, the
// fast reciprocal (within 2 ulp).  (A correctly rounded reciprocal by FMA steps
// from the hardware estimate has the division's bits and is slower: its steps
// follow one another.  Bit-exact sweeps x, y, z in us, FMA steps / division:
// SP 128x128x16 163, 162, 98 / 157, 154, 94; BT 304x208x17 2271, 1777, 1252 /
// 2258, 1762, 1241.)
template <typename T>
__device__ __forceinline__ T pivot_recip(T b) { return NPBMZ_HAS_FP32 ? nr_rcp(b) : (T)1.0 / b; }
template <>
__device__ __forceinline__ float pivot_recip<float>(float b) { return __fdividef(1.0f, b); }

#if NPBMZ_HAS_FP32
#include "bt_lines.cuh"
#else
// Columns of C that are nonzero in pivot row p when it is reached: the block's
// own, and all once the row of the normal momentum (all nonzero) has been the
// pivot; the other columns hold exact zeros, whose operations are skipped.
template <int DIR>
__host__ __device__ constexpr bool cfull(int p, int c) {
  if (p > DIR + 1) return true;
  for (int q = 0; q <= p; ++q)
    if (anz<DIR>(q, c)) return true;
  return false;
}

// binvcrhs (src/BT/solve_subs.jl:468-723): Gauss-Jordan on B, no pivoting,
// applied to C and r.
template <int DIR>
__device__ __forceinline__ void binvcrhs(double B[5][5], double C[5][5], double r[5]) {
#pragma unroll
  for (int p = 0; p < 5; ++p) {
    const double pivot = pivot_recip<double>(B[p][p]);
#pragma unroll
    for (int c = p + 1; c < 5; ++c) B[p][c] *= pivot;
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (cfull<DIR>(p, c)) C[p][c] *= pivot;
    r[p] *= pivot;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (q == p) continue;
      const double coeff = B[q][p];
#pragma unroll
      for (int c = p + 1; c < 5; ++c) B[q][c] -= coeff * B[p][c];
#pragma unroll
      for (int c = 0; c < 5; ++c)
        if (cfull<DIR>(p, c)) C[q][c] -= coeff * C[p][c];
      r[q] -= coeff * r[p];
    }
  }
}

template <int DIR>
__device__ __forceinline__ void bt_load_point(const Fields& F, int64_t pt, double& ri, double& u2, double& u3,
                                              double& u4, double& u5, double& q) {
  const int64_t NP = F.NP;
  ri = F.prim[PR_RHOI * NP + pt];
  q = F.prim[PR_QS * NP + pt];
  u2 = F.u[NP + pt];
  u3 = F.u[2 * NP + pt];
  u4 = F.u[3 * NP + pt];
  u5 = F.u[4 * NP + pt];
}

template <int DIR>
__global__ void __launch_bounds__(128) k_bt_solve(Fields F, Consts K, const Work* __restrict__ work,
                                                  double* __restrict__ lhsc, int64_t nlt, int add_u) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  double* __restrict__ rhs = F.rhs;

  const double tmp1 = DIR == 0 ? K.dttx1 : DIR == 1 ? K.dtty1 : K.dttz1;
  const double tmp2 = DIR == 0 ? K.dttx2 : DIR == 1 ? K.dtty2 : K.dttz2;
  const double dd[5] = {DIR == 0 ? K.dx1 : DIR == 1 ? K.dy1 : K.dz1, DIR == 0 ? K.dx2 : DIR == 1 ? K.dy2 : K.dz2,
                        DIR == 0 ? K.dx3 : DIR == 1 ? K.dy3 : K.dz3, DIR == 0 ? K.dx4 : DIR == 1 ? K.dy4 : K.dz4,
                        DIR == 0 ? K.dx5 : DIR == 1 ? K.dy5 : K.dz5};

  double rp[5];          // r' at p-1
  double Cp[5][5];       // C' at p-1
  double Acur[5][5];     // lhsa at p   (structural nonzeros only)
  double Anext[5][5];    // lhsa at p+1
  double Bcur[5][5];     // lhsb at p   (structural nonzeros only)
  double f[5][5], nj[5][5];
  double ri, u2, u3, u4, u5, q;

#pragma unroll
  for (int m = 0; m < 5; ++m) rp[m] = rhs[m * NP + base];
  // Jacobian at point 0 -> lhsa at 1; at point 1 -> lhsb at 1 and lhsa at 2.
  bt_load_point<DIR>(F, base, ri, u2, u3, u4, u5, q);
  bt_jac<DIR>(K, ri, u2, u3, u4, u5, q, f, nj);
  bt_scale<DIR>(f, nj, tmp1, tmp2);
  bt_asm_a<DIR>(f, nj, tmp1, dd, Acur);
  bt_load_point<DIR>(F, base + st, ri, u2, u3, u4, u5, q);
  bt_jac<DIR>(K, ri, u2, u3, u4, u5, q, f, nj);
  bt_scale<DIR>(f, nj, tmp1, tmp2);
  bt_asm_b(nj, tmp1, dd, Bcur);
  if (n - 2 >= 2) bt_asm_a<DIR>(f, nj, tmp1, dd, Anext);

  for (int p = 1; p <= n - 2; ++p) {
    const int64_t pt = base + p * st;
    double r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = rhs[m * NP + pt];
    // matvec_sub(lhsa_p, r'_{p-1}, r_p): the row sum is formed first.
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double s;
      bool have = false;
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        if (!anz<DIR>(m, c)) continue;
        s = have ? s + Acur[m][c] * rp[c] : Acur[m][c] * rp[c];
        have = true;
      }
      r[m] -= s;
    }
    // lhsb_p (full) = lhsb_p - lhsa_p * C'_{p-1}, one term at a time; C'_0 = 0.
    double B[5][5];
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        double t = bnz(a, b) ? Bcur[a][b] : 0.0;
        bool have = bnz(a, b);
        if (p > 1) {
#pragma unroll
          for (int c = 0; c < 5; ++c) {
            if (!anz<DIR>(a, c)) continue;
            t = have ? t - Acur[a][c] * Cp[c][b] : -(Acur[a][c] * Cp[c][b]);
            have = true;
          }
        }
        B[a][b] = t;
      }
    // Jacobian at p+1 -> lhsc_p, lhsb_{p+1}, lhsa_{p+2}
    bt_load_point<DIR>(F, pt + st, ri, u2, u3, u4, u5, q);
    bt_jac<DIR>(K, ri, u2, u3, u4, u5, q, f, nj);
    bt_scale<DIR>(f, nj, tmp1, tmp2);
    double C[5][5];
    bt_asm_c<DIR>(f, nj, tmp1, dd, C);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b)
        if (anz<DIR>(a, b)) Acur[a][b] = Anext[a][b];
    if (p + 1 <= n - 2) bt_asm_b(nj, tmp1, dd, Bcur);
    if (p + 2 <= n - 2) bt_asm_a<DIR>(f, nj, tmp1, dd, Anext);
    binvcrhs<DIR>(B, C, r);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        Cp[a][b] = C[a][b];
        lhsc[((int64_t)p * 25 + a * 5 + b) * nlt + gl] = C[a][b];
      }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      rp[m] = r[m];
      rhs[m * NP + pt] = r[m];
    }
  }
  // back substitution: r_p -= C'_p r_{p+1}, one term at a time; the boundary
  // value r_{n-1} is unchanged by the forward sweep.
  double rn[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) rn[m] = rhs[m * NP + base + (n - 1) * st];
  for (int p = n - 2; p >= 1; --p) {
    const int64_t pt = base + p * st;
    double r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = (p == n - 2) ? rp[m] : rhs[m * NP + pt];
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
      for (int c = 0; c < 5; ++c) r[m] -= lhsc[((int64_t)p * 25 + m * 5 + c) * nlt + gl] * rn[c];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double v = r[m];
      rhs[m * NP + pt] = v;
      if (add_u) F.u[m * NP + pt] += v;
      rn[m] = r[m];
    }
  }
}

#endif  // NPBMZ_HAS_FP32

#if NPBMZ_HAS_FP32
// ============================================================================
// Mixed-precision BT sweep (NPBMZ_MIXED): two kernels per sweep direction.
//
// Pass 1 (k_bt_mixed_solve): T x0 = b in FP32 from the FP32 state copies,
// C' and the forward-eliminated rhs kept as FP32 in the line scratch
// (30 floats per point), x0 written as FP32.
// Pass 2 (k_bt_refine): the residual r = b - T x0 in FP64, T d = r in FP32,
// x = x0 + d into rhs (and, after the z sweep, into u).  Row p of T applied
// to x is, with F_q = fjac_q x_q and N_q = njac_q x_q,
//   x_p + tmp2 (F_{p+1} - F_{p-1}) - tmp1 (N_{p-1} - 2 N_p + N_{p+1})
//       - tmp1 D (x_{p-1} - 2 x_p + x_{p+1})
// (lhsa/lhsb/lhsc of src/BT/x_solve.jl:613-708 applied to x), and F, N are
// formed from the velocities directly (bt_jx), so the FP64 work is about
// 90 operations per point.  Boundary rows are identity rows whose residual
// is exactly zero, so d = 0 there.
// ============================================================================
template <int DIR>
__device__ __forceinline__ void bt_jx(const Consts& K, double ri, double q, double u2, double u3, double u4, double u5,
                                      const double x[5], double Fx[5], double Nx[5]) {
  const double vel[3] = {u2 * ri, u3 * ri, u4 * ri};
  const double E = u5 * ri;
  constexpr int a = DIR + 1;  // the momentum component normal to the sweep
  const double vn = vel[DIR];
  const double c1 = K.c1, c2 = K.c2;
  double d[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) d[m] = x[m + 1] - vel[m] * x[0];
  double tang = 0.0;
  Fx[0] = x[a];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    if (m == DIR) continue;
    Fx[m + 1] = vn * d[m] + vel[m] * x[a];
    tang += vel[m] * x[m + 1];
  }
  Fx[a] = (c2 * q - vn * vn) * x[0] - c2 * tang + (2.0 - c2) * vn * x[a] + c2 * x[4];
  Fx[4] = (2.0 * c2 * q - c1 * E) * vn * x[0] - c2 * vn * tang + (c1 * E - c2 * (q + vn * vn)) * x[a] + c1 * vn * x[4];
  const double k43 = K.con43 * K.c3c4, c3c4 = K.c3c4, c1345 = K.c1345;
  double s4 = c1345 * (x[4] - E * x[0]);
  Nx[0] = 0.0;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double cm = (m == DIR) ? k43 : c3c4;
    Nx[m + 1] = cm * ri * d[m];
    s4 += (cm - c1345) * vel[m] * d[m];
  }
  Nx[4] = ri * s4;
}

// State of the FP32 block elimination carried from point p to p+1.
template <int DIR>
struct BtF32Carry {
  float Cp[5][5];     // C' at p-1
  float rp[5];        // forward-eliminated rhs at p-1
  float Pcur[5][5];   // -lhsa at p   (structural nonzeros)
  float Pnext[5][5];  // -lhsa at p+1
  float Bs[5][5];     // lhsb at p    (structural nonzeros)
};

constexpr int BT_SCR = 30;  // words per point of the FP32 line scratch: C' (25), r' (5)

// G and H from the FP32 state s = ri, u2, u3, u4, u5, q.
template <int DIR>
__device__ __forceinline__ void bt_gh_f32(const BtK<float>& k, const float s[6], BtGH<DIR, float>& J) {
  const float v[3] = {s[1] * s[0], s[2] * s[0], s[3] * s[0]};
  bt_gh<DIR, float>(k, s[0], v, s[4] * s[0], s[5], J);
}

// Start of the elimination: Jacobians at points 0 and 1 (FP32 state s0, s1).
template <int DIR>
__device__ __forceinline__ void bt_f32_begin(const BtK<float>& k, const float s0[6], const float s1[6],
                                             BtF32Carry<DIR>& c) {
  BtGH<DIR, float> J;
  bt_gh_f32<DIR>(k, s0, J);
  bt_form_p<DIR, float>(J, c.Pcur);
  bt_gh_f32<DIR>(k, s1, J);
  bt_form_p<DIR, float>(J, c.Pnext);
  bt_form_b<DIR, float>(J, c.Bs);
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) c.Cp[a][b] = 0.f;
}

// One forward step at point p (1..n-2): r holds the rhs of row p on entry and
// the eliminated rhs on exit; sn is the FP32 state at p+1.  C'_p (STORE_C)
// and r'_p go to out[e * nlt] (the point's words of the line scratch).
template <int DIR, bool STORE_C>
__device__ __forceinline__ void bt_f32_step(const BtK<float>& k, float r[5], const float sn[6], BtF32Carry<DIR>& c,
                                            float* __restrict__ out, int64_t nlt) {
  float B[5][5], C[5][5];
  BtGH<DIR, float> J;
  bt_add_px<DIR, float>(c.Pcur, c.rp, r);
  bt_add_pc<DIR, float>(c.Pcur, c.Cp, c.Bs, B);
  bt_gh_f32<DIR>(k, sn, J);
  bt_form_c<DIR, float>(J, C);
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b)
      if (anz<DIR>(a, b)) c.Pcur[a][b] = c.Pnext[a][b];
  bt_form_p<DIR, float>(J, c.Pnext);
  bt_form_b<DIR, float>(J, c.Bs);
  bt_factor_solve<DIR, float>(B, C, r);
#pragma unroll
  for (int a = 0; a < 5; ++a)
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      c.Cp[a][b] = C[a][b];
      if (STORE_C) out[(a * 5 + b) * nlt] = C[a][b];
    }
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    c.rp[m] = r[m];
    out[(25 + m) * nlt] = r[m];
  }
}

__device__ __forceinline__ void load_state_f32(const Fields& F, int64_t pt, float s[6]) {
  const int64_t NP = F.NP;
  s[0] = F.primf[PF_RHOI * NP + pt];
  s[1] = F.primf[PF_U2 * NP + pt];
  s[2] = F.primf[PF_U3 * NP + pt];
  s[3] = F.primf[PF_U4 * NP + pt];
  s[4] = F.primf[PF_U5 * NP + pt];
  s[5] = F.primf[PF_QS * NP + pt];
}

__device__ __forceinline__ void load_state_f64(const Fields& F, int64_t pt, double s[6]) {
  const int64_t NP = F.NP;
  s[0] = F.prim[PR_RHOI * NP + pt];
  s[1] = F.u[NP + pt];
  s[2] = F.u[2 * NP + pt];
  s[3] = F.u[3 * NP + pt];
  s[4] = F.u[4 * NP + pt];
  s[5] = F.prim[PR_QS * NP + pt];
}

// Pass 1: T x0 = b in FP32.  Loads of point p+2 and of b_{p+1} are issued one
// step ahead so that they overlap the elimination of point p.
template <int DIR>
__device__ __forceinline__ void bt_mixed_item(const Fields& F, const Consts& K, const Work w, float* __restrict__ scr,
                                              int64_t nlt, float* __restrict__ x0) {
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  const double* __restrict__ rhs = F.rhs;
  auto bload = [&](int m, int64_t pt) -> float { return (float)rhs[m * NP + pt]; };
  BtF32Carry<DIR> c;
  float s0[6], s1[6];
  load_state_f32(F, base, s0);
  load_state_f32(F, base + st, s1);
#pragma unroll
  for (int m = 0; m < 5; ++m) c.rp[m] = bload(m, base);
  bt_f32_begin<DIR>(bt_consts<float>(K, DIR), s0, s1, c);
  float sn[6], bn[5];
  load_state_f32(F, base + 2 * st, sn);
#pragma unroll
  for (int m = 0; m < 5; ++m) bn[m] = bload(m, base + st);
  for (int p = 1; p <= n - 2; ++p) {
    float r[5], s[6];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = bn[m];
#pragma unroll
    for (int e = 0; e < 6; ++e) s[e] = sn[e];
    if (p + 1 <= n - 2) {  // prefetch for the next step
      load_state_f32(F, base + (int64_t)(p + 2) * st, sn);
#pragma unroll
      for (int m = 0; m < 5; ++m) bn[m] = bload(m, base + (int64_t)(p + 1) * st);
    }
    bt_f32_step<DIR, true>(bt_consts<float>(K, DIR), r, s, c, scr + (int64_t)p * BT_SCR * nlt + gl, nlt);
  }
  float rn[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) rn[m] = bload(m, base + (int64_t)(n - 1) * st);
  for (int p = n - 2; p >= 1; --p) {
    float r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = (p == n - 2) ? c.rp[m] : scr[((int64_t)p * BT_SCR + 25 + m) * nlt + gl];
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
      for (int cc = 0; cc < 5; ++cc) r[m] -= scr[((int64_t)p * BT_SCR + m * 5 + cc) * nlt + gl] * rn[cc];
    const int64_t pt = base + p * st;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      x0[m * NP + pt] = r[m];
      rn[m] = r[m];
    }
  }
}

template <int DIR>
__global__ void __launch_bounds__(128) k_bt_mixed_solve(Fields F, Consts K, const Work* __restrict__ work, int nwork,
                                                        float* __restrict__ scr, int64_t nlt, float* __restrict__ x0) {
  for (int it = blockIdx.x; it < nwork; it += gridDim.x) bt_mixed_item<DIR>(F, K, work[it], scr, nlt, x0);
}

// Pass 2: r = b - T x0 in FP64, T d = r in FP32, x = x0 + d.  The residual
// rows are accumulated point by point: point q adds
//   -tmp2 F_q - tmp1 N_q - tmp1 D x_q          to row q+1,
//   x_q + 2 tmp1 N_q + 2 tmp1 D x_q            to row q,
//   tmp2 F_q - tmp1 N_q - tmp1 D x_q           to row q-1 (which is then complete).
template <int DIR>
__global__ void __launch_bounds__(128) k_bt_refine(Fields F, Consts K, const Work* __restrict__ work,
                                                   float* __restrict__ scr, int64_t nlt, int add_u,
                                                   const float* __restrict__ x0f) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  double* __restrict__ rhs = F.rhs;

  const double t1d = DIR == 0 ? K.dttx1 : DIR == 1 ? K.dtty1 : K.dttz1;
  const double t2d = DIR == 0 ? K.dttx2 : DIR == 1 ? K.dtty2 : K.dttz2;
  double ddd[5];
  if (DIR == 0) { ddd[0] = K.dx1; ddd[1] = K.dx2; ddd[2] = K.dx3; ddd[3] = K.dx4; ddd[4] = K.dx5; }
  else if (DIR == 1) { ddd[0] = K.dy1; ddd[1] = K.dy2; ddd[2] = K.dy3; ddd[3] = K.dy4; ddd[4] = K.dy5; }
  else { ddd[0] = K.dz1; ddd[1] = K.dz2; ddd[2] = K.dz3; ddd[3] = K.dz4; ddd[4] = K.dz5; }

  // x0 at point q: the FP32 first pass inside, b itself on the boundary.
  auto load_x = [&](int q, double x[5]) {
    const int64_t pt = base + (int64_t)q * st;
    if (q == 0 || q == n - 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = rhs[m * NP + pt];
    } else {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = (double)x0f[m * NP + pt];
    }
  };
  double acc_c[5], acc_n[5];   // partial (T x0) of rows p and p+1
  double xq[5], sq[6];
  float s0[6], s1[6];
  // point 0: contributes to row 1 only (row 0 is an identity row)
  load_x(0, xq);
  load_state_f64(F, base, sq);
  {
    double Fq[5], Nq[5];
    bt_jx<DIR>(K, sq[0], sq[5], sq[1], sq[2], sq[3], sq[4], xq, Fq, Nq);
#pragma unroll
    for (int m = 0; m < 5; ++m) acc_c[m] = -t2d * Fq[m] - t1d * Nq[m] - t1d * ddd[m] * xq[m];
#pragma unroll
    for (int e = 0; e < 6; ++e) s0[e] = (float)sq[e];
  }
  // point 1: centre of row 1, left neighbour of row 2
  load_x(1, xq);
  load_state_f64(F, base + st, sq);
  {
    double Fq[5], Nq[5];
    bt_jx<DIR>(K, sq[0], sq[5], sq[1], sq[2], sq[3], sq[4], xq, Fq, Nq);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      acc_c[m] += xq[m] + 2.0 * t1d * Nq[m] + 2.0 * t1d * ddd[m] * xq[m];
      acc_n[m] = -t2d * Fq[m] - t1d * Nq[m] - t1d * ddd[m] * xq[m];
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) s1[e] = (float)sq[e];
  }
  BtF32Carry<DIR> c;
#pragma unroll
  for (int m = 0; m < 5; ++m) c.rp[m] = 0.f;  // the boundary residual is exactly zero
  bt_f32_begin<DIR>(bt_consts<float>(K, DIR), s0, s1, c);
  // prefetch point 2 and b_1
  double xn[5], sn[6], bn[5];
  load_x(2, xn);
  load_state_f64(F, base + 2 * st, sn);
#pragma unroll
  for (int m = 0; m < 5; ++m) bn[m] = rhs[m * NP + base + st];

  for (int p = 1; p <= n - 2; ++p) {
    const int64_t pt = base + (int64_t)p * st;
    double b[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) { xq[m] = xn[m]; b[m] = bn[m]; }
#pragma unroll
    for (int e = 0; e < 6; ++e) sq[e] = sn[e];
    if (p + 1 <= n - 2) {
      load_x(p + 2, xn);
      load_state_f64(F, base + (int64_t)(p + 2) * st, sn);
#pragma unroll
      for (int m = 0; m < 5; ++m) bn[m] = rhs[m * NP + base + (int64_t)(p + 1) * st];
    }
    // point p+1 completes row p
    double Fq[5], Nq[5];
    bt_jx<DIR>(K, sq[0], sq[5], sq[1], sq[2], sq[3], sq[4], xq, Fq, Nq);
    float r[5], s[6];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double tx = acc_c[m] + t2d * Fq[m] - t1d * Nq[m] - t1d * ddd[m] * xq[m];
      r[m] = (float)(b[m] - tx);
      acc_c[m] = acc_n[m] + xq[m] + 2.0 * t1d * Nq[m] + 2.0 * t1d * ddd[m] * xq[m];
      acc_n[m] = -t2d * Fq[m] - t1d * Nq[m] - t1d * ddd[m] * xq[m];
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) s[e] = (float)sq[e];
    bt_f32_step<DIR, true>(bt_consts<float>(K, DIR), r, s, c, scr + (int64_t)p * BT_SCR * nlt + gl, nlt);
    (void)pt;
  }
  // back substitution of the correction d, then x = x0 + d
  float dn[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (int p = n - 2; p >= 1; --p) {
    const int64_t pt = base + p * st;
    float d[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) d[m] = (p == n - 2) ? c.rp[m] : scr[((int64_t)p * BT_SCR + 25 + m) * nlt + gl];
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
      for (int cc = 0; cc < 5; ++cc) d[m] -= scr[((int64_t)p * BT_SCR + m * 5 + cc) * nlt + gl] * dn[cc];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double v = (double)x0f[m * NP + pt] + (double)d[m];
      rhs[m * NP + pt] = v;
      if (add_u) F.u[m * NP + pt] += v;
      dn[m] = d[m];
    }
  }
}

// ============================================================================
// Double-float (FP32 pair) arithmetic for the residual of the refinement
// pass.  GB300 issues FP32 at 64x the FP64 rate; a value hi + lo with
// |lo| <= ulp(hi)/2 carries about 48 significant bits, enough for the
// residual r = b - T x0 (its error enters the refined solution at about
// 1e-14 relative, below the FP32 re-solve's own (eps32 * kappa)^2 term).
// Error-free transformations (Knuth two-sum, FMA two-product) are written
// with explicit round-to-nearest intrinsics so no contraction or
// reassociation can change them.
// ============================================================================
struct df64 {
  float hi, lo;
};

__device__ __forceinline__ df64 df_quick(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ df64 df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ df64 df_add(df64 a, df64 b) {
  const df64 s = df_two_sum(a.hi, b.hi);
  return df_quick(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ df64 df_neg(df64 a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ df64 df_sub(df64 a, df64 b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ df64 df_mul(df64 a, df64 b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return df_quick(p, e);
}
__device__ __forceinline__ df64 df_scale2(df64 a) { return {2.f * a.hi, 2.f * a.lo}; }  // exact
__device__ __forceinline__ df64 f2df(float2 v) { return {v.x, v.y}; }
// FP32 -> FP64 (exact) from the bit pattern: sign, exponent rebiased by
// 1023 - 127, significand shifted into place; zero, subnormals, inf and nan
// take the conversion instruction, which on GB300 is an FP64-pipe slot.
__device__ __forceinline__ double f32_to_f64(float f) {
  const unsigned b = __float_as_uint(f);
  const unsigned e = (b >> 23) & 0xffu;
  if (e - 1u >= 254u) return (double)f;
  const unsigned hi = (b & 0x80000000u) | ((e + 896u) << 20) | ((b >> 3) & 0xfffffu);
  return __hiloint2double((int)hi, (int)(b << 29));
}
__device__ __forceinline__ double df_to_double(df64 v) { return f32_to_f64(v.hi) + f32_to_f64(v.lo); }
// 1/a: FP32 estimate x, residual e = 1 - a x formed exactly to first order
// (a.hi x = p + pe exactly; 1 - p is exact since p is within 2^-23 of 1),
// then x + x e.
__device__ __forceinline__ df64 df_rcp(df64 a) {
  const float x = __frcp_rn(a.hi);
  const float p = __fmul_rn(a.hi, x);
  const float pe = __fmaf_rn(a.hi, x, -p);
  const float e = __fmaf_rn(-a.lo, x, __fsub_rn(__fsub_rn(1.f, p), pe));
  return df_quick(x, __fmul_rn(x, e));
}
__device__ __forceinline__ float2 df2f(df64 v) { return make_float2(v.hi, v.lo); }
__device__ __forceinline__ df64 df_from(double d) {
  const float h = __double2float_rn(d);
  return {h, __double2float_rn(d - (double)h)};
}

// The same without renormalisation: the residual's sums and products.  The low
// word of a sum is bounded by its summands, 2^-23 of the largest, not by the sum:
// after a cancellation it may be as large as the high word.  So are the errors,
// as those of the normalised forms are (the residual is judged by its terms'
// size): a sum rounds its low word twice, 2^-46 of the largest summand.  A
// product rounds its low word as much and drops the low words' product: with one
// operand a sum, the other's low word is within 2^-23 of it (a pair, a product,
// or none: plain FP32), which is 2^-46 again; with both operands sums nothing
// bounds a low word by its high one, and du_mul_ss keeps their product.  That is
// 4 or 5 operations instead of 7, 8 instead of 11 for a sum.
// With the plain FP32 operands the residual takes 640 instructions a point
// instead of 1040 (480x320x28 sweeps 586, 568, 635 -> 550, 527, 582 us); u's
// error against 64 bits after 20 steps of 64x64x8 is 2.8e-15 (before 3.5e-15),
// after 10 of 480x320x28 1.3e-15 (1.5e-15).
__device__ __forceinline__ df64 du_mul(df64 a, df64 b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  return {p, __fmaf_rn(a.lo, b.hi, e)};
}
__device__ __forceinline__ df64 du_mul_ss(df64 a, df64 b) {  // both operands sums
  const df64 r = du_mul(a, b);
  return {r.hi, __fmaf_rn(a.lo, b.lo, r.lo)};
}
__device__ __forceinline__ df64 du_add(df64 a, df64 b) {
  const df64 s = df_two_sum(a.hi, b.hi);
  return {s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo))};
}
__device__ __forceinline__ df64 du_sub(df64 a, df64 b) { return du_add(a, df_neg(b)); }
// with a plain FP32 operand: the first pass's solution inside the line
__device__ __forceinline__ df64 du_mul(df64 a, float b) {
  const float p = __fmul_rn(a.hi, b);
  return {p, __fmaf_rn(a.lo, b, __fmaf_rn(a.hi, b, -p))};
}
__device__ __forceinline__ df64 du_add(df64 a, float b) {
  const df64 s = df_two_sum(a.hi, b);
  return {s.hi, __fadd_rn(s.lo, a.lo)};
}

// Constants of the residual in one direction (pairs); t2 carries the sign of
// the direction the line is walked in.
struct BtResid {
  df64 t1, t2, t1d[5], c1, c2, two_m_c2, k43, c3c4, c1345, k43m, c3c4m;
};
template <int DIR>
__device__ __forceinline__ BtResid bt_resid_consts(const Consts& K, bool turned) {
  BtResid c;
  c.t1 = f2df(K.p_dtt1[DIR]);
  c.t2 = f2df(K.p_dtt2[DIR]);
  if (turned) c.t2 = df_neg(c.t2);
#pragma unroll
  for (int m = 0; m < 5; ++m) c.t1d[m] = f2df(K.p_t1d[DIR][m]);
  c.c1 = f2df(K.p_c1);
  c.c2 = f2df(K.p_c2);
  c.two_m_c2 = f2df(K.p_two_m_c2);
  c.k43 = f2df(K.p_k43);
  c.c3c4 = f2df(K.p_c3c4);
  c.c1345 = f2df(K.p_c1345);
  c.k43m = f2df(K.p_k43m);
  c.c3c4m = f2df(K.p_c3c4m);
  return c;
}

// P = tmp2 fjac x and Q = tmp1 (njac + D) x of one point (the formulas of
// bt_jx); X = float inside the line, df64 at its ends.
template <int DIR, typename X>
__device__ __forceinline__ void bt_pq(const BtResid& k, const df64 st[6], const X x[5], df64 P[5], df64 Q[5]) {
  // st = ri, u2, u3, u4, u5, q
  const df64 ri = st[0], q = st[5];
  const df64 vel[3] = {du_mul(st[1], ri), du_mul(st[2], ri), du_mul(st[3], ri)};
  const df64 E = du_mul(st[4], ri);
  constexpr int a = DIR + 1, m1 = DIR == 0 ? 1 : 0, m2 = DIR == 2 ? 1 : 2;
  const df64 vn = vel[DIR];
  df64 d[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) d[m] = du_add(df_neg(du_mul(vel[m], x[0])), x[m + 1]);
  df64 Fx[5];
#pragma unroll
  for (int m = 0; m < 3; ++m)
    if (m != DIR) Fx[m + 1] = du_add(du_mul_ss(vn, d[m]), du_mul(vel[m], x[a]));
  const df64 tang = du_add(du_mul(vel[m1], x[m1 + 1]), du_mul(vel[m2], x[m2 + 1]));
  const df64 c2q = du_mul(k.c2, q), vn2 = du_mul(vn, vn), c1E = du_mul(k.c1, E);
  Fx[a] = du_add(du_sub(du_mul(du_sub(c2q, vn2), x[0]), du_mul(k.c2, tang)),
                 du_add(du_mul(du_mul(k.two_m_c2, vn), x[a]), du_mul(k.c2, x[4])));
  Fx[4] = du_add(du_sub(du_mul(du_mul_ss(du_sub(df_scale2(c2q), c1E), vn), x[0]), du_mul_ss(du_mul(k.c2, vn), tang)),
                 du_add(du_mul(du_sub(c1E, du_mul(k.c2, du_add(q, vn2))), x[a]), du_mul(du_mul(k.c1, vn), x[4])));
  df64 s4 = du_mul(k.c1345, du_add(df_neg(du_mul(E, x[0])), x[4]));
  const df64 k43ri = du_mul(k.k43, ri), c3c4ri = du_mul(k.c3c4, ri);
  P[0] = du_mul(k.t2, x[a]);
  Q[0] = du_mul(k.t1d[0], x[0]);
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    Q[m + 1] = du_add(du_mul(k.t1, du_mul_ss(m == DIR ? k43ri : c3c4ri, d[m])), du_mul(k.t1d[m + 1], x[m + 1]));
    s4 = du_add(s4, du_mul_ss(du_mul(m == DIR ? k.k43m : k.c3c4m, vel[m]), d[m]));
  }
  Q[4] = du_add(du_mul(k.t1, du_mul_ss(ri, s4)), du_mul(k.t1d[4], x[4]));
#pragma unroll
  for (int m = 1; m < 5; ++m) P[m] = du_mul(k.t2, Fx[m]);
}

__device__ __forceinline__ void load_state_df(const Fields& F, int64_t pt, df64 s[6]) {
  const int64_t NP = F.NP;
  const int order[6] = {PF_RHOI, PF_U2, PF_U3, PF_U4, PF_U5, PF_QS};
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    s[e].hi = F.primf[order[e] * NP + pt];
    s[e].lo = F.primf[(PF_HI_COUNT + order[e]) * NP + pt];
  }
}

// Refinement pass with the residual in double-float.  Point q contributes,
// with P_q = tmp2 F_q and Q_q = tmp1 (N_q + D x_q),
//   -P_q - Q_q to row q+1,   x_q + 2 Q_q to row q,   P_q - Q_q to row q-1.
template <int DIR>
__global__ void __launch_bounds__(128) k_bt_refine_df(Fields F, Consts K, const Work* __restrict__ work,
                                                      float* __restrict__ scr, int64_t nlt, int add_u,
                                                      const float* __restrict__ x0f) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  double* __restrict__ rhs = F.rhs;
  const BtResid kr = bt_resid_consts<DIR>(K, false);
  auto load_x = [&](int q, df64 x[5]) {
    const int64_t pt = base + (int64_t)q * st;
    if (q == 0 || q == n - 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = df_from(rhs[m * NP + pt]);
    } else {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = {x0f[m * NP + pt], 0.f};
    }
  };
  df64 acc_c[5], acc_n[5], xq[5], sq[6], P[5], Q[5];
  float s0[6], s1[6];
  load_x(0, xq);
  load_state_df(F, base, sq);
  bt_pq<DIR>(kr, sq, xq, P, Q);
#pragma unroll
  for (int m = 0; m < 5; ++m) acc_c[m] = df_neg(df_add(P[m], Q[m]));
#pragma unroll
  for (int e = 0; e < 6; ++e) s0[e] = sq[e].hi;
  load_x(1, xq);
  load_state_df(F, base + st, sq);
  bt_pq<DIR>(kr, sq, xq, P, Q);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    acc_c[m] = df_add(acc_c[m], df_add(xq[m], df_scale2(Q[m])));
    acc_n[m] = df_neg(df_add(P[m], Q[m]));
  }
#pragma unroll
  for (int e = 0; e < 6; ++e) s1[e] = sq[e].hi;
  BtF32Carry<DIR> c;
#pragma unroll
  for (int m = 0; m < 5; ++m) c.rp[m] = 0.f;
  // bt_f32_begin takes ri, u2, u3, u4, u5, q in that order (as sq)
  bt_f32_begin<DIR>(bt_consts<float>(K, DIR), s0, s1, c);
  df64 xn[5], sn[6];
  double bn[5];  // b of the next point
  auto load_b = [&](int64_t pt) {
#pragma unroll
    for (int m = 0; m < 5; ++m) bn[m] = rhs[m * NP + pt];
  };
  load_x(2, xn);
  load_state_df(F, base + 2 * st, sn);
  load_b(base + st);

  for (int p = 1; p <= n - 2; ++p) {
    double b[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      xq[m] = xn[m];
      b[m] = bn[m];
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) sq[e] = sn[e];
    if (p + 1 <= n - 2) {
      load_x(p + 2, xn);
      load_state_df(F, base + (int64_t)(p + 2) * st, sn);
      load_b(base + (int64_t)(p + 1) * st);
    }
    bt_pq<DIR>(kr, sq, xq, P, Q);
    float r[5], s[6];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const df64 tx = df_add(acc_c[m], df_sub(P[m], Q[m]));
      r[m] = __double2float_rn((b[m] - (double)tx.hi) - (double)tx.lo);
      acc_c[m] = df_add(acc_n[m], df_add(xq[m], df_scale2(Q[m])));
      acc_n[m] = df_neg(df_add(P[m], Q[m]));
    }
#pragma unroll
    for (int e = 0; e < 6; ++e) s[e] = sq[e].hi;
    bt_f32_step<DIR, true>(bt_consts<float>(K, DIR), r, s, c, scr + (int64_t)p * BT_SCR * nlt + gl, nlt);
  }
  float dn[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (int p = n - 2; p >= 1; --p) {
    const int64_t pt = base + p * st;
    float d[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) d[m] = (p == n - 2) ? c.rp[m] : scr[((int64_t)p * BT_SCR + 25 + m) * nlt + gl];
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
      for (int cc = 0; cc < 5; ++cc) d[m] -= scr[((int64_t)p * BT_SCR + m * 5 + cc) * nlt + gl] * dn[cc];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double v = (double)x0f[m * NP + pt] + (double)d[m];
      rhs[m * NP + pt] = v;
      if (add_u) F.u[m * NP + pt] += v;
      dn[m] = d[m];
    }
  }
}

// ============================================================================
// Software-pipelined refined FP32 BT sweep of a fused step (mode 4).
// Each thread streams its data PIPE points ahead with cp.async into a ring of
// PIPE slots in shared memory (word e of slot s of thread t at
// ring[(s * W + e) * T + t]: a warp's copies land in consecutive banks), in
// the forward elimination and in the back substitution alike.
//
// TWO: two threads per line, eliminating from both ends: thread t of the first
// half of the block takes rows 1..L0 of its line from point 0 up, thread
// t + lines the rows n-2..L0+1 from point n-1 down (L0 = (n-1)/2 rows, L1 the
// rest).  Seen from the far end the line is the same one with the sign of the
// convective terms turned (G -> -G: lhsa and lhsc trade places), so both
// halves run the same code on a local index j, q = j or n-1-j.  At the seam
//   x_A = r'_A - C'_A x_B,  x_B = r'_B - C'_B x_A
// (A, B the two middle rows), so each half solves (I - C'_A C'_B) x_A =
// r'_A - C'_A r'_B with its partner's C' and r' and substitutes back toward
// its own end.  A line then takes half as many dependent steps for 8 % more
// instructions and a barrier: faster while the lines are too few to fill the
// chip one per thread (few_lines in npbmz_api.cu draws the line).
// ============================================================================
#ifndef NPBMZ_PIPE
#define NPBMZ_PIPE 4
#endif
constexpr int PIPE = NPBMZ_PIPE;

// Minimum resident CTAs of 128 threads per SM that the pipelined sweep
// kernels are compiled for (__launch_bounds__): it caps their registers at
// 65536 / (128 * n) and so sets their occupancy.
#ifndef NPBMZ_BT_MIXED_MINB
#define NPBMZ_BT_MIXED_MINB 1
#endif
#ifndef NPBMZ_BT_REFINE_MINB
#define NPBMZ_BT_REFINE_MINB 1
#endif
#ifndef NPBMZ_SP_MINB
#define NPBMZ_SP_MINB 3
#endif

__device__ __forceinline__ void cpa4(float* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa8(double* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr int PL_MIXED_W = 30;   // words per slot, first pass
constexpr int PL_REFINE_W = 45;  // words per slot, refinement pass
// Words per thread beside the ring: at the seam C' and r' (TWO), else b at the
// line's last point in double-float.
__host__ __device__ constexpr int pl_end_words(bool two) { return two ? 30 : 10; }

// Dynamic shared memory of the pipelined kernels for tpb lines per block.
__host__ __device__ constexpr size_t pl_mixed_smem(int tpb, bool two) {
  return (size_t)(PIPE * PL_MIXED_W + pl_end_words(two)) * (two ? 2 : 1) * tpb * sizeof(float);
}
__host__ __device__ constexpr size_t pl_refine_smem(int tpb, bool two) {
  return (size_t)(PIPE * PL_REFINE_W + pl_end_words(two)) * (two ? 2 : 1) * tpb * sizeof(float);
}

// A thread's part of a line (TWO: one half): local point j is point q(j).
template <int DIR, bool TWO>
struct BtHalf {
  int n, L;           // points of the line, rows of this half
  bool far;           // the half that starts at point n-1
  bool active;        // the block's last lines may be missing
  int64_t base, st, gl;
  __device__ __forceinline__ int q(int j) const { return TWO && far ? n - 1 - j : j; }
  __device__ __forceinline__ int64_t pt(int j) const { return base + (int64_t)q(j) * st; }
};
template <int DIR, bool TWO>
__device__ __forceinline__ BtHalf<DIR, TWO> bt_half(const ZoneDev& Z, int first) {
  BtHalf<DIR, TWO> h;
  const int lines = TWO ? blockDim.x >> 1 : blockDim.x;
  h.far = TWO && (int)threadIdx.x >= lines;
  const int line = first + (int)threadIdx.x - (h.far ? lines : 0);
  h.active = line < zone_lines(Z, DIR);
  h.n = zone_line_len(Z, DIR);
  const int L0 = TWO ? (h.n - 1) >> 1 : h.n - 2;
  h.L = h.far ? h.n - 2 - L0 : L0;
  if (h.active) line_geometry(Z, DIR, line, h.base, h.st);
  h.gl = Z.lineoff[DIR] + line;
  return h;
}

// The direction's constants with the sign of the convective terms turned for
// the far half.
template <int DIR>
__device__ __forceinline__ BtK<float> bt_half_consts(const Consts& K, bool far) {
  BtK<float> k = bt_consts<float>(K, DIR);
  if (far) {
    k.t2 = -k.t2;
    k.c2t2 = -k.c2t2;
    k.c1t2 = -k.c1t2;
  }
  return k;
}

// The seam: x of this half's last row from its own and its partner's C', r'
// (join: 30 words per thread).  All threads of the block call it.
__device__ __forceinline__ void bt_join(float* join, bool far, const float C[5][5], const float r[5], float x[5]) {
  const int T = blockDim.x, lines = T >> 1, t = threadIdx.x, u = far ? t - lines : t + lines;
#pragma unroll
  for (int e = 0; e < 25; ++e) join[e * T + t] = C[e / 5][e % 5];
#pragma unroll
  for (int m = 0; m < 5; ++m) join[(25 + m) * T + t] = r[m];
  __syncthreads();
  float M[5][5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    x[m] = r[m];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      x[m] = fmaf(-C[m][c], join[(25 + c) * T + u], x[m]);
      M[m][c] = m == c ? 1.f : 0.f;
    }
  }
#pragma unroll
  for (int e = 0; e < 5; ++e)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const float b = join[(e * 5 + c) * T + u];
#pragma unroll
      for (int m = 0; m < 5; ++m) M[m][c] = fmaf(-C[m][e], b, M[m][c]);
    }
#pragma unroll
  for (int p = 0; p < 5; ++p) {
    const float piv = bt_recip(M[p][p]);
#pragma unroll
    for (int c = p + 1; c < 5; ++c) M[p][c] *= piv;
    x[p] *= piv;
#pragma unroll
    for (int q = p + 1; q < 5; ++q) {
#pragma unroll
      for (int c = p + 1; c < 5; ++c) M[q][c] = fmaf(-M[q][p], M[p][c], M[q][c]);
      x[q] = fmaf(-M[q][p], x[p], x[q]);
    }
  }
#pragma unroll
  for (int p = 4; p > 0; --p)
#pragma unroll
    for (int q = 0; q < p; ++q) x[q] = fmaf(-M[q][p], x[p], x[q]);
  __syncthreads();  // join may be written again (the block's next item)
}

template <int DIR, bool TWO>
__device__ __forceinline__ void bt_mixed_pl_item(const Fields& F, const Consts& K, const Work w,
                                                 float* __restrict__ scr, int64_t nlt, float* __restrict__ x0,
                                                 unsigned char* pl_smem) {
  const ZoneDev Z = F.zones[w.zone];
  const BtHalf<DIR, TWO> h = bt_half<DIR, TWO>(Z, w.first);
  if (!TWO && !h.active) return;
  const int64_t NP = F.NP;
  const int T = blockDim.x, L = h.L;
  float* my = reinterpret_cast<float*>(pl_smem) + threadIdx.x;
  auto S = [&](int slot, int e) -> float* { return my + (slot * PL_MIXED_W + e) * T; };
  const int order[6] = {PF_RHOI, PF_U2, PF_U3, PF_U4, PF_U5, PF_QS};
  // the x sweep reads its x-line-major copies, y and z the zone layout
  auto st_at = [&](int j, int plane) -> const float* {
    return DIR == 0 ? F.pfx + ((int64_t)h.q(j) * PF_COUNT + plane) * F.nlx + h.gl : F.primf + plane * NP + h.pt(j);
  };
  auto b_at = [&](int j, int e) -> const float* {
    return DIR == 0 ? F.rdx + ((int64_t)h.q(j) * 10 + e) * F.nlx + h.gl : F.rdf + e * NP + h.pt(j);
  };
  auto x0_at = [&](int j, int m) -> float* {
    return DIR == 0 ? F.x0x + ((int64_t)h.q(j) * 5 + m) * F.nlx + h.gl : x0 + m * NP + h.pt(j);
  };
  auto scr_at = [&](int j, int e) -> float* { return scr + ((int64_t)h.q(j) * BT_SCR + e) * nlt + h.gl; };
  // forward step j (1..L) consumes b_j and the state at j+1
  auto issue_fwd = [&](int j) {
    if (j <= L) {
      const int slot = j % PIPE;
#pragma unroll
      for (int e = 0; e < 6; ++e) cpa4(S(slot, e), st_at(j + 1, order[e]));
#pragma unroll
      for (int m = 0; m < 5; ++m) cpa4(S(slot, 6 + m), b_at(j, m));
    }
    cpa_commit();
  };
  const BtK<float> k = bt_half_consts<DIR>(K, h.far);
  BtF32Carry<DIR> c;
  float* ends = reinterpret_cast<float*>(pl_smem) + (size_t)PIPE * PL_MIXED_W * T;
  if (h.active) {
    // the ring's first slots (and b at the last point, which a whole line's
    // back substitution starts from) go out before the line's first points
    // are read directly, so that the memory latencies overlap
    if (!TWO) {
#pragma unroll
      for (int m = 0; m < 5; ++m) cpa4(ends + m * T + threadIdx.x, b_at(h.n - 1, m));
    }
#pragma unroll
    for (int j = 1; j < PIPE; ++j) issue_fwd(j);
    {
      float s0[6], s1[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        s0[e] = *st_at(0, order[e]);
        s1[e] = *st_at(1, order[e]);
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) c.rp[m] = *b_at(0, m);
      bt_f32_begin<DIR>(k, s0, s1, c);
    }
    for (int j = 1; j <= L; ++j) {
      issue_fwd(j + PIPE - 1);
      cpa_wait<PIPE - 1>();
      const int slot = j % PIPE;
      float r[5], s[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) s[e] = *S(slot, e);
#pragma unroll
      for (int m = 0; m < 5; ++m) r[m] = *S(slot, 6 + m);
      bt_f32_step<DIR, true>(k, r, s, c, scr_at(j, 0), nlt);
      if (j + PIPE > L) {
        // the ring does not refill this slot: C'_j and r'_j stay here for the
        // back substitution, which so starts without a trip to memory
#pragma unroll
        for (int a = 0; a < 5; ++a)
#pragma unroll
          for (int b = 0; b < 5; ++b) *S(slot, a * 5 + b) = c.Cp[a][b];
#pragma unroll
        for (int m = 0; m < 5; ++m) *S(slot, 25 + m) = c.rp[m];
      }
    }
    cpa_wait<0>();
  }
  float rn[5];
  if (TWO) {
    bt_join(ends, h.far, c.Cp, c.rp, rn);
    if (!h.active) return;
  } else {
#pragma unroll
    for (int m = 0; m < 5; ++m) rn[m] = ends[m * T + threadIdx.x];
  }
  // back substitution (TWO: row L is the seam's): step j consumes C'_j and
  // r'_j from slot j % PIPE: the last PIPE rows as the forward pass left
  // them, the others loaded PIPE steps ahead into the slot just consumed
  auto issue_bwd = [&](int j) {
    if (j >= 1) {
      const int slot = j % PIPE;
#pragma unroll
      for (int e = 0; e < 30; ++e) cpa4(S(slot, e), scr_at(j, e));
    }
    cpa_commit();
  };
  for (int j = L; j >= 1; --j) {
    if (j + PIPE <= L) cpa_wait<PIPE - 1>();
    const int slot = j % PIPE;
    if (!TWO || j < L) {
      float r[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float t = *S(slot, 25 + m);
#pragma unroll
        for (int cc = 0; cc < 5; ++cc) t -= *S(slot, m * 5 + cc) * rn[cc];
        r[m] = t;
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) rn[m] = r[m];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) *x0_at(j, m) = rn[m];
    issue_bwd(j - PIPE);
  }
  cpa_wait<0>();
}

template <int DIR, bool TWO>
__global__ void __launch_bounds__(TWO ? 256 : 128, NPBMZ_BT_MIXED_MINB) k_bt_mixed_pl(Fields F, Consts K, const Work* __restrict__ work, int nwork,
                                                     float* __restrict__ scr, int64_t nlt, float* __restrict__ x0) {
  extern __shared__ __align__(16) unsigned char pl_smem[];
  for (int it = blockIdx.x; it < nwork; it += gridDim.x) bt_mixed_pl_item<DIR, TWO>(F, K, work[it], scr, nlt, x0, pl_smem);
}

template <int DIR, bool OUT_DF, bool TWO>
__device__ __forceinline__ void bt_refine_pl_item(const Fields& F, const Consts& K, const Work w,
                                                  float* __restrict__ scr, int64_t nlt, int add_u,
                                                  const float* __restrict__ x0f, unsigned char* pl_smem) {
  const ZoneDev Z = F.zones[w.zone];
  const BtHalf<DIR, TWO> h = bt_half<DIR, TWO>(Z, w.first);
  if (!TWO && !h.active) return;
  const int64_t NP = F.NP;
  const int T = blockDim.x, L = h.L;
  float* my = reinterpret_cast<float*>(pl_smem) + threadIdx.x;
  auto S = [&](int slot, int e) -> float* { return my + (slot * PL_REFINE_W + e) * T; };
  double* __restrict__ rhs = F.rhs;
  float* __restrict__ bdf = F.rdf;
  const int order[6] = {PF_RHOI, PF_U2, PF_U3, PF_U4, PF_U5, PF_QS};
  // the x sweep reads its x-line-major copies, y and z the zone layout; the
  // result always goes to the zone layout (the next sweep reads it there)
  auto st_at = [&](int j, int plane) -> const float* {
    return DIR == 0 ? F.pfx + ((int64_t)h.q(j) * PF_COUNT + plane) * F.nlx + h.gl : F.primf + plane * NP + h.pt(j);
  };
  auto b_at = [&](int j, int e) -> float* {
    return DIR == 0 ? F.rdx + ((int64_t)h.q(j) * 10 + e) * F.nlx + h.gl : bdf + e * NP + h.pt(j);
  };
  auto x0_at = [&](int j, int m) -> const float* {
    return DIR == 0 ? F.x0x + ((int64_t)h.q(j) * 5 + m) * F.nlx + h.gl : x0f + m * NP + h.pt(j);
  };
  auto scr_at = [&](int j, int e) -> float* { return scr + ((int64_t)h.q(j) * BT_SCR + e) * nlt + h.gl; };

  const BtResid kr = bt_resid_consts<DIR>(K, h.far);
  // x at local point j: b itself at the line's ends, else the first pass's
  auto load_x = [&](int j, df64 x[5]) {
#pragma unroll
    for (int m = 0; m < 5; ++m)
      x[m] = (j == 0 || j == h.n - 1) ? df64{*b_at(j, m), *b_at(j, 5 + m)} : df64{*x0_at(j, m), 0.f};
  };
  auto load_sdf = [&](int j, df64 s6[6]) {
#pragma unroll
    for (int e = 0; e < 6; ++e) s6[e] = df64{*st_at(j, order[e]), *st_at(j, PF_HI_COUNT + order[e])};
  };
  // forward step j (1..L) consumes x0 and the state at j+1 and b_j: words
  // 0..4 x0, 5..16 state hi/lo, 17..26 b hi/lo
  auto issue_fwd = [&](int j) {
    if (j <= L) {
      const int slot = j % PIPE;
      if (j + 1 < h.n - 1) {
#pragma unroll
        for (int m = 0; m < 5; ++m) cpa4(S(slot, m), x0_at(j + 1, m));
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        cpa4(S(slot, 5 + e), st_at(j + 1, order[e]));
        cpa4(S(slot, 11 + e), st_at(j + 1, PF_HI_COUNT + order[e]));
      }
#pragma unroll
      for (int e = 0; e < 10; ++e) cpa4(S(slot, 17 + e), b_at(j, e));
    }
    cpa_commit();
  };
  // back substitution step j consumes C'_j (the first pass's), r'_j, x0_j and
  // u_j: words 0..24, 25..29, 30..34, 35..44 (u in two halves)
  auto fetch_bwd = [&](int j, bool r_in_slot) {
    const int slot = j % PIPE;
#pragma unroll
    for (int e = 0; e < 30; ++e)
      if (e < 25 || !r_in_slot) cpa4(S(slot, e), scr_at(j, e));
#pragma unroll
    for (int m = 0; m < 5; ++m) cpa4(S(slot, 30 + m), x0_at(j, m));
    if (!OUT_DF && add_u) {
      const float* up = reinterpret_cast<const float*>(F.u + h.pt(j));
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        cpa4(S(slot, 35 + 2 * m), up + 2 * m * NP);
        cpa4(S(slot, 36 + 2 * m), up + 2 * m * NP + 1);
      }
    }
  };
  const BtK<float> k = bt_half_consts<DIR>(K, h.far);
  BtF32Carry<DIR> c;
  float* ends = reinterpret_cast<float*>(pl_smem) + (size_t)PIPE * PL_REFINE_W * T;
  if (h.active) {
    // the ring's first slots (and x at a whole line's last point, b itself) go
    // out before the line's first points are read directly, so that the
    // memory latencies overlap
    if (!TWO) {
#pragma unroll
      for (int e = 0; e < 10; ++e) cpa4(ends + e * T + threadIdx.x, b_at(h.n - 1, e));
    }
#pragma unroll
    for (int j = 1; j < PIPE; ++j) issue_fwd(j);
    // partial sums of T x0: rows j and j + 1
    df64 acc_c[5], acc_n[5], sq[6], P[5], Q[5];
    {
      float s0[6], s1[6];
      df64 xe[5];
      load_x(0, xe);
      load_sdf(0, sq);
      bt_pq<DIR>(kr, sq, xe, P, Q);
#pragma unroll
      for (int m = 0; m < 5; ++m) acc_c[m] = df_neg(du_add(P[m], Q[m]));
#pragma unroll
      for (int e = 0; e < 6; ++e) s0[e] = sq[e].hi;
      load_x(1, xe);
      load_sdf(1, sq);
      bt_pq<DIR>(kr, sq, xe, P, Q);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        acc_c[m] = du_add(acc_c[m], du_add(df_scale2(Q[m]), xe[m]));
        acc_n[m] = df_neg(du_add(P[m], Q[m]));
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) s1[e] = sq[e].hi;
#pragma unroll
      for (int m = 0; m < 5; ++m) c.rp[m] = 0.f;
      bt_f32_begin<DIR>(k, s0, s1, c);
    }
    for (int j = 1; j <= L; ++j) {
      issue_fwd(j + PIPE - 1);
      cpa_wait<PIPE - 1>();
      const int slot = j % PIPE;
      df64 bd[5];
      float r[5], s[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) sq[e] = df64{*S(slot, 5 + e), *S(slot, 11 + e)};
#pragma unroll
      for (int m = 0; m < 5; ++m) bd[m] = df64{*S(slot, 17 + m), *S(slot, 22 + m)};
#pragma unroll
      for (int e = 0; e < 6; ++e) s[e] = sq[e].hi;
      if (j + 1 < h.n - 1) {
        float xq[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) xq[m] = *S(slot, m);
        bt_pq<DIR>(kr, sq, xq, P, Q);
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          const df64 rr = du_sub(bd[m], du_add(acc_c[m], du_sub(P[m], Q[m])));
          r[m] = rr.hi + rr.lo;
          acc_c[m] = du_add(acc_n[m], du_add(df_scale2(Q[m]), xq[m]));
          acc_n[m] = df_neg(du_add(P[m], Q[m]));
        }
      } else {  // the line's last point: completes the last row
        df64 xe[5];
        if (TWO) {  // a line of one row
          load_x(j + 1, xe);
        } else {
#pragma unroll
          for (int m = 0; m < 5; ++m) xe[m] = df64{ends[m * T + threadIdx.x], ends[(5 + m) * T + threadIdx.x]};
        }
        bt_pq<DIR>(kr, sq, xe, P, Q);
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          const df64 rr = du_sub(bd[m], du_add(acc_c[m], du_sub(P[m], Q[m])));
          r[m] = rr.hi + rr.lo;
        }
      }
      // the elimination runs again: its factors would be 25 more words a point
      // to write and read (480x320x28 x, y, z 640, 610, 681 -> 821, 901, 918 us);
      // C' is the first pass's, so only r' is stored
      bt_f32_step<DIR, false>(k, r, s, c, scr_at(j, 0), nlt);
      if (j + PIPE > L) {
        // the ring does not refill this slot: r'_j stays here for the back
        // substitution, whose other operands are fetched now, so that it
        // starts without a trip to memory
#pragma unroll
        for (int m = 0; m < 5; ++m) *S(slot, 25 + m) = r[m];
        fetch_bwd(j, true);
        cpa_commit();
      }
    }
  }
  float dn[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  if (TWO) {
    bt_join(ends, h.far, c.Cp, c.rp, dn);
    if (!h.active) return;
  }
  cpa_wait<0>();
  // back substitution (TWO: row L is the seam's): step j from slot
  // j % PIPE: the last PIPE rows as the forward pass left them, the others
  // fetched PIPE steps ahead into the slot just consumed
  for (int j = L; j >= 1; --j) {
    if (j + PIPE <= L) cpa_wait<PIPE - 1>();
    const int slot = j % PIPE;
    const int64_t pt = h.pt(j);
    if (!TWO || j < L) {
      float d[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float t = *S(slot, 25 + m);
#pragma unroll
        for (int cc = 0; cc < 5; ++cc) t -= *S(slot, m * 5 + cc) * dn[cc];
        d[m] = t;
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) dn[m] = d[m];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const float xv = *S(slot, 30 + m);
      if (OUT_DF) {
        // x: in place of b in the x-line-major copy (k_xline_back moves it
        // to rdf); y: rdf
        const df64 v = df_two_sum(xv, dn[m]);
        *b_at(j, m) = v.hi;
        *b_at(j, 5 + m) = v.lo;
      } else {
        // exact FP32 -> FP64 by bits (a conversion instruction takes the FP64 pipe)
        const double v = f32_to_f64(xv) + f32_to_f64(dn[m]);
        rhs[m * NP + pt] = v;
        if (add_u)
          F.u[m * NP + pt] = __hiloint2double(__float_as_int(*S(slot, 36 + 2 * m)), __float_as_int(*S(slot, 35 + 2 * m))) + v;
      }
    }
    if (j - PIPE >= 1) fetch_bwd(j - PIPE, false);
    cpa_commit();
  }
  cpa_wait<0>();
}

template <int DIR, bool OUT_DF, bool TWO>
__global__ void __launch_bounds__(TWO ? 256 : 128, NPBMZ_BT_REFINE_MINB) k_bt_refine_pl(Fields F, Consts K, const Work* __restrict__ work, int nwork,
                                                      float* __restrict__ scr, int64_t nlt, int add_u,
                                                      const float* __restrict__ x0f) {
  extern __shared__ __align__(16) unsigned char pl_smem[];
  for (int it = blockIdx.x; it < nwork; it += gridDim.x)
    bt_refine_pl_item<DIR, OUT_DF, TWO>(F, K, work[it], scr, nlt, add_u, x0f, pl_smem);
}
#endif  // NPBMZ_HAS_FP32

// ============================================================================
// SP scalar pentadiagonal line solve, one thread per line.
// lhsx / lhsy / lhsz assembly (src/SP/lhsx.jl:27-111, lhsy.jl, lhsz.jl), the
// Thomas forward elimination and back substitution (src/SP/x_solve.jl:203-313,
// 456-512; y_solve.jl, z_solve.jl), then ninvr / pinvr / tzetar
// (src/SP/ninvr.jl:19-32, pinvr.jl:20-33, tzetar.jl:27-52) and, after the z
// sweep, add (src/SP/add.jl:14-23).  Rows 0 and n-1 are the identity rows
// lhsinit leaves in the persistent lhs (src/SP/initialize.jl:235-256); they go
// through the same elimination as in the reference.  The bands l4, l5 of each
// of the 3 systems are kept for the back substitution in
// scr[(p*6 + b) * nlt + global_line].
// ============================================================================
struct SpBands {
  double l[3][5];
};

template <int DIR, typename T, typename G>
__device__ __forceinline__ void sp_assemble(const Consts& K, int q, int n, const G cv[3], const G rhon[3],
                                            const G spd[3], T L[3][5]) {
  if (q == 0 || q == n - 1) {
#pragma unroll
    for (int s = 0; s < 3; ++s) { L[s][0] = (T)0.0; L[s][1] = (T)0.0; L[s][2] = (T)1.0; L[s][3] = (T)0.0; L[s][4] = (T)0.0; }
    return;
  }
  const G dtt1 = kv<G>(DIR == 0 ? K.dttx1 : DIR == 1 ? K.dtty1 : K.dttz1, K.f_dtt1[DIR]);
  const G dtt2 = kv<G>(DIR == 0 ? K.dttx2 : DIR == 1 ? K.dtty2 : K.dttz2, K.f_dtt2[DIR]);
  const G c2dtt1 = kv<G>(DIR == 0 ? K.c2dttx1 : DIR == 1 ? K.c2dtty1 : K.c2dttz1, K.f_c2dtt1[DIR]);
  const G comz1 = kv<G>(K.comz1, K.f_comz1), comz4 = kv<G>(K.comz4, K.f_comz4);
  const G comz5 = kv<G>(K.comz5, K.f_comz5), comz6 = kv<G>(K.comz6, K.f_comz6);
  G L1 = (G)0.0;
  G L2 = -dtt2 * cv[0] - dtt1 * rhon[0];
  G L3 = (G)1.0 + c2dtt1 * rhon[1];
  G L4 = dtt2 * cv[2] - dtt1 * rhon[2];
  G L5 = (G)0.0;
  if (q == 1) { L3 += comz5; L4 -= comz4; L5 += comz1; }
  if (q == 2) { L2 -= comz4; L3 += comz6; L4 -= comz4; L5 += comz1; }
  if (q >= 3 && q <= n - 4) { L1 += comz1; L2 -= comz4; L3 += comz6; L4 -= comz4; L5 += comz1; }
  if (q == n - 3) { L1 += comz1; L2 -= comz4; L3 += comz6; L4 -= comz4; }
  if (q == n - 2) { L1 += comz1; L2 -= comz4; L3 += comz5; }
  L[0][0] = (T)L1; L[0][1] = (T)L2; L[0][2] = (T)L3; L[0][3] = (T)L4; L[0][4] = (T)L5;
  L[1][0] = (T)L1; L[1][1] = (T)(L2 - dtt2 * spd[0]); L[1][2] = (T)L3; L[1][3] = (T)(L4 + dtt2 * spd[2]); L[1][4] = (T)L5;
  L[2][0] = (T)L1; L[2][1] = (T)(L2 + dtt2 * spd[0]); L[2][2] = (T)L3; L[2][3] = (T)(L4 - dtt2 * spd[2]); L[2][4] = (T)L5;
}

template <int DIR>
__device__ __forceinline__ void sp_geom(const Fields& F, const Consts& K, int64_t pt, double& cv, double& rhon,
                                        double& spd) {
  const int64_t NP = F.NP;
  const double ru1 = K.c3c4 * F.prim[PR_RHOI * NP + pt];
  cv = F.prim[(DIR == 0 ? PR_US : DIR == 1 ? PR_VS : PR_WS) * NP + pt];
  const double da = DIR == 0 ? K.dx2 : DIR == 1 ? K.dy3 : K.dz4;
  const double db = DIR == 0 ? K.dx5 : DIR == 1 ? K.dy5 : K.dz5;
  const double dm = DIR == 0 ? K.dxmax : DIR == 1 ? K.dymax : K.dzmax;
  const double dc = DIR == 0 ? K.dx1 : DIR == 1 ? K.dy1 : K.dz1;
  rhon = fmax(fmax(fmax(da + K.con43 * ru1, db + K.c1c5 * ru1), dm + ru1), dc);
  spd = F.prim[PR_SPEED * NP + pt];
}

// system s covers rhs components [s==0 ? 0..2 : s==1 ? 3 : 4]
#define SP_M0(s) ((s) == 0 ? 0 : (s) + 2)
#define SP_M1(s) ((s) == 0 ? 2 : (s) + 2)

// out / transform: the in-place solve writes the transformed solution into
// rhs (out == rhs, transform = 1); the first pass of the refined solve writes
// the untransformed solution of the interior points to a separate buffer.
template <int DIR, typename T>
__global__ void __launch_bounds__(128) k_sp_solve(Fields F, Consts K, const Work* __restrict__ work,
                                                  T* __restrict__ scr, int64_t nlt, int add_u,
                                                  double* __restrict__ out, int transform) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  double* __restrict__ rhs = F.rhs;

  // geometry window for assembling row q: values at q-1, q, q+1
  double gcv[4], grh[4], gsp[4];   // values at rows a-1 .. a+2 of a sliding window
  T cur3[3], cur4[3], cur5[3];     // row p   (l3, l4, l5), modified
  T nx2[3], nx3[3], nx4[3], nx5[3];  // row p+1 (l2..l5), modified
  T rr[3][5];                       // rhs rows p, p+1, p+2

  // rows 0 and 1: assemble
  {
    T L0[3][5], L1[3][5];
    double cv[3], rh[3], sp[3];
    // row 0 is an identity row; its geometry is not needed.
    sp_assemble<DIR, T>(K, 0, n, cv, rh, sp, L0);
    sp_geom<DIR>(F, K, base, gcv[0], grh[0], gsp[0]);
    sp_geom<DIR>(F, K, base + st, gcv[1], grh[1], gsp[1]);
    sp_geom<DIR>(F, K, base + 2 * st, gcv[2], grh[2], gsp[2]);
    cv[0] = gcv[0]; cv[1] = gcv[1]; cv[2] = gcv[2];
    rh[0] = grh[0]; rh[1] = grh[1]; rh[2] = grh[2];
    sp[0] = gsp[0]; sp[1] = gsp[1]; sp[2] = gsp[2];
    sp_assemble<DIR, T>(K, 1, n, cv, rh, sp, L1);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      cur3[s] = L0[s][2]; cur4[s] = L0[s][3]; cur5[s] = L0[s][4];
      nx2[s] = L1[s][1]; nx3[s] = L1[s][2]; nx4[s] = L1[s][3]; nx5[s] = L1[s][4];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      rr[0][m] = (T)rhs[m * NP + base];
      rr[1][m] = (T)rhs[m * NP + base + st];
    }
  }
  // window gcv[0..2] now holds rows 0,1,2.
  for (int p = 0; p <= n - 3; ++p) {
    // assemble row p+2 (needs geometry at p+1, p+2, p+3)
    T L2[3][5];
    {
      double cv[3], rh[3], sp[3];
      const int q = p + 2;
      if (q + 1 <= n - 1) sp_geom<DIR>(F, K, base + (int64_t)(q + 1) * st, gcv[3], grh[3], gsp[3]);
      cv[0] = gcv[1]; cv[1] = gcv[2]; cv[2] = gcv[3];
      rh[0] = grh[1]; rh[1] = grh[2]; rh[2] = grh[3];
      sp[0] = gsp[1]; sp[1] = gsp[2]; sp[2] = gsp[3];
      sp_assemble<DIR, T>(K, q, n, cv, rh, sp, L2);
      gcv[0] = gcv[1]; gcv[1] = gcv[2]; gcv[2] = gcv[3];
      grh[0] = grh[1]; grh[1] = grh[2]; grh[2] = grh[3];
      gsp[0] = gsp[1]; gsp[1] = gsp[2]; gsp[2] = gsp[3];
    }
    const int64_t pt2 = base + (int64_t)(p + 2) * st;
#pragma unroll
    for (int m = 0; m < 5; ++m) rr[2][m] = (T)rhs[m * NP + pt2];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const T fac1 = pivot_recip<T>(cur3[s]);
      cur4[s] *= fac1;
      cur5[s] *= fac1;
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[0][m] *= fac1;
      nx3[s] -= nx2[s] * cur4[s];
      nx4[s] -= nx2[s] * cur5[s];
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] -= nx2[s] * rr[0][m];
      T n2 = L2[s][1], n3 = L2[s][2];
      n2 -= L2[s][0] * cur4[s];
      n3 -= L2[s][0] * cur5[s];
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[2][m] -= L2[s][0] * rr[0][m];
      scr[((int64_t)p * 6 + 2 * s) * nlt + gl] = cur4[s];
      scr[((int64_t)p * 6 + 2 * s + 1) * nlt + gl] = cur5[s];
      // shift the window: row p+1 becomes current, row p+2 next
      cur3[s] = nx3[s]; cur4[s] = nx4[s]; cur5[s] = nx5[s];
      nx2[s] = n2; nx3[s] = n3; nx4[s] = L2[s][3]; nx5[s] = L2[s][4];
    }
    const int64_t pt = base + (int64_t)p * st;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      if (p > 0) out[m * NP + pt] = (double)rr[0][m];
      rr[0][m] = rr[1][m];
      rr[1][m] = rr[2][m];
    }
  }
  // last two rows: p = n-2 (current), n-1 (next)
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const T fac1 = pivot_recip<T>(cur3[s]);
    cur4[s] *= fac1;
    cur5[s] *= fac1;
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[0][m] *= fac1;
    nx3[s] -= nx2[s] * cur4[s];
    nx4[s] -= nx2[s] * cur5[s];
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] -= nx2[s] * rr[0][m];
    const T fac2 = pivot_recip<T>(nx3[s]);
    nx4[s] *= fac2;
    nx5[s] *= fac2;
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] *= fac2;
  }
  // back substitution; rr[0] = row n-2, rr[1] = row n-1 (the boundary row,
  // numerically unchanged).  b1 = r_{p+1}, b2 = r_{p+2} before transforms.
  T b1[5], b2[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) b2[m] = rr[1][m];
  {
    const int p = n - 2;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int s = m < 3 ? 0 : m - 2;
      b1[m] = rr[0][m] - cur4[s] * b2[m];
    }
    (void)p;
  }
  // Emit row n-2, then rows n-3 .. 1.
  auto emit = [&](int p, const T v[5]) {
    const int64_t pt = base + (int64_t)p * st;
    double r1 = (double)v[0], r2 = (double)v[1], r3 = (double)v[2], r4 = (double)v[3], r5 = (double)v[4];
    if (!transform) {
      out[pt] = r1; out[NP + pt] = r2; out[2 * NP + pt] = r3; out[3 * NP + pt] = r4; out[4 * NP + pt] = r5;
      return;
    }
    double o[5];
    if (DIR == 0) {  // ninvr
      const double t1 = K.bt * r3;
      const double t2 = 0.5e0 * (r4 + r5);
      o[0] = -r2; o[1] = r1; o[2] = K.bt * (r4 - r5); o[3] = -t1 + t2; o[4] = t1 + t2;
    } else if (DIR == 1) {  // pinvr
      const double t1 = K.bt * r1;
      const double t2 = 0.5e0 * (r4 + r5);
      o[0] = K.bt * (r4 - r5); o[1] = -r3; o[2] = r2; o[3] = -t1 + t2; o[4] = t1 + t2;
    } else {  // tzetar
      const double xvel = F.prim[PR_US * NP + pt], yvel = F.prim[PR_VS * NP + pt], zvel = F.prim[PR_WS * NP + pt];
      const double ac = F.prim[PR_SPEED * NP + pt], acinv = F.prim[PR_AINV * NP + pt];
      const double ac2u = ac * ac;
      const double uzik1 = F.u[pt];
      const double btuz = K.bt * uzik1;
      const double t1 = btuz * acinv * (r4 + r5);
      const double t2 = r3 + t1;
      const double t3 = btuz * (r4 - r5);
      o[0] = t2;
      o[1] = -uzik1 * r2 + xvel * t2;
      o[2] = uzik1 * r1 + yvel * t2;
      o[3] = zvel * t2 + t3;
      o[4] = uzik1 * (-xvel * r2 + yvel * r1) + F.prim[PR_QS * NP + pt] * t2 + K.c2iv * ac2u * t1 + zvel * t3;
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      rhs[m * NP + pt] = o[m];
      if (add_u) F.u[m * NP + pt] += o[m];
    }
  };
  // row n-2's transform must read u before row n-2 is updated; emit updates
  // only its own point, so the order below is safe.
  emit(n - 2, b1);
  for (int p = n - 3; p >= 1; --p) {
    const int64_t pt = base + (int64_t)p * st;
    T r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int s = m < 3 ? 0 : m - 2;
      const T l4 = scr[((int64_t)p * 6 + 2 * s) * nlt + gl];
      const T l5 = scr[((int64_t)p * 6 + 2 * s + 1) * nlt + gl];
      r[m] = (T)out[m * NP + pt];
      r[m] -= l4 * b1[m] + l5 * b2[m];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) { b2[m] = b1[m]; b1[m] = r[m]; }
    emit(p, r);
  }
}

// ============================================================================
// Refinement pass of the mixed-precision SP sweep: residual r = b - L x0 of
// each scalar pentadiagonal system in FP64 (bands of lhsx/lhsy/lhsz
// assembled in FP64), FP32 Thomas solve of L d = r, x = x0 + d, then the
// sweep's transform (ninvr / pinvr / tzetar) and, after the z sweep, add.
// x0 comes from xw on interior points; boundary rows are identity rows, so
// x0 there is b itself and the residual is zero.
// ============================================================================
template <int DIR>
__device__ __forceinline__ void sp_transform(const Fields& F, const Consts& K, int64_t pt, const double v[5],
                                             double o[5]) {
  const int64_t NP = F.NP;
  const double r1 = v[0], r2 = v[1], r3 = v[2], r4 = v[3], r5 = v[4];
  if (DIR == 0) {
    const double t1 = K.bt * r3;
    const double t2 = 0.5e0 * (r4 + r5);
    o[0] = -r2; o[1] = r1; o[2] = K.bt * (r4 - r5); o[3] = -t1 + t2; o[4] = t1 + t2;
  } else if (DIR == 1) {
    const double t1 = K.bt * r1;
    const double t2 = 0.5e0 * (r4 + r5);
    o[0] = K.bt * (r4 - r5); o[1] = -r3; o[2] = r2; o[3] = -t1 + t2; o[4] = t1 + t2;
  } else {
    const double xvel = F.prim[PR_US * NP + pt], yvel = F.prim[PR_VS * NP + pt], zvel = F.prim[PR_WS * NP + pt];
    const double ac = F.prim[PR_SPEED * NP + pt], acinv = F.prim[PR_AINV * NP + pt];
    const double ac2u = ac * ac;
    const double uzik1 = F.u[pt];
    const double btuz = K.bt * uzik1;
    const double t1 = btuz * acinv * (r4 + r5);
    const double t2 = r3 + t1;
    const double t3 = btuz * (r4 - r5);
    o[0] = t2;
    o[1] = -uzik1 * r2 + xvel * t2;
    o[2] = uzik1 * r1 + yvel * t2;
    o[3] = zvel * t2 + t3;
    o[4] = uzik1 * (-xvel * r2 + yvel * r1) + F.prim[PR_QS * NP + pt] * t2 + K.c2iv * ac2u * t1 + zvel * t3;
  }
}

// Geometry of one point for the SP band assembly, generic in the type.
template <int DIR, typename G>
__device__ __forceinline__ void sp_geom_t(G ri, G cvel, G spd_in, const Consts& K, G& cv, G& rhon, G& spd) {
  const G ru1 = kv<G>(K.c3c4, K.f_c3c4) * ri;
  cv = cvel;
  const G da = kv<G>(DIR == 0 ? K.dx2 : DIR == 1 ? K.dy3 : K.dz4, K.f_d[DIR][DIR + 1]);
  const G db = kv<G>(DIR == 0 ? K.dx5 : DIR == 1 ? K.dy5 : K.dz5, K.f_d[DIR][4]);
  const G dm = kv<G>(DIR == 0 ? K.dxmax : DIR == 1 ? K.dymax : K.dzmax, K.f_dmax[DIR]);
  const G dc = kv<G>(DIR == 0 ? K.dx1 : DIR == 1 ? K.dy1 : K.dz1, K.f_d[DIR][0]);
  rhon = fmax(fmax(fmax(da + kv<G>(K.con43, K.f_con43) * ru1, db + kv<G>(K.c1c5, K.f_c1c5) * ru1), dm + ru1), dc);
  spd = spd_in;
}

// Thomas forward elimination of the three SP systems over one line, in FP32,
// with rows supplied by row_at(q, L, r) (q = 0..n-1; L[3][5] bands, r[5]).
// Bands l4, l5 and the eliminated rhs of rows 0..n-3 go to the line scratch
// scr[(p*11 + e) * nlt + gl]; rows n-2 and n-1 stay in the returned state.
struct SpF32Tail {
  float cur4[3];     // l4 of row n-2
  float r2[5];       // eliminated rhs of row n-2
  float rlast[5];    // eliminated rhs of row n-1
};

template <typename RowAt>
__device__ __forceinline__ void sp_forward_f32(int n, float* __restrict__ scr, int64_t nlt, int64_t gl, RowAt row_at,
                                               SpF32Tail& tail) {
  float cur3[3], cur4[3], cur5[3], nx2[3], nx3[3], nx4[3], nx5[3];
  float rr[3][5];
  {
    float L0[3][5], L1[3][5];
    row_at(0, L0, rr[0]);
    row_at(1, L1, rr[1]);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      cur3[s] = L0[s][2]; cur4[s] = L0[s][3]; cur5[s] = L0[s][4];
      nx2[s] = L1[s][1]; nx3[s] = L1[s][2]; nx4[s] = L1[s][3]; nx5[s] = L1[s][4];
    }
  }
  for (int p = 0; p <= n - 3; ++p) {
    float L2[3][5];
    row_at(p + 2, L2, rr[2]);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const float fac1 = __fdividef(1.0f, cur3[s]);
      cur4[s] *= fac1;
      cur5[s] *= fac1;
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[0][m] *= fac1;
      nx3[s] -= nx2[s] * cur4[s];
      nx4[s] -= nx2[s] * cur5[s];
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] -= nx2[s] * rr[0][m];
      float n2 = L2[s][1], n3 = L2[s][2];
      n2 -= L2[s][0] * cur4[s];
      n3 -= L2[s][0] * cur5[s];
#pragma unroll
      for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[2][m] -= L2[s][0] * rr[0][m];
      scr[((int64_t)p * 11 + 2 * s) * nlt + gl] = cur4[s];
      scr[((int64_t)p * 11 + 2 * s + 1) * nlt + gl] = cur5[s];
      cur3[s] = nx3[s]; cur4[s] = nx4[s]; cur5[s] = nx5[s];
      nx2[s] = n2; nx3[s] = n3; nx4[s] = L2[s][3]; nx5[s] = L2[s][4];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      scr[((int64_t)p * 11 + 6 + m) * nlt + gl] = rr[0][m];
      rr[0][m] = rr[1][m];
      rr[1][m] = rr[2][m];
    }
  }
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const float fac1 = __fdividef(1.0f, cur3[s]);
    cur4[s] *= fac1;
    cur5[s] *= fac1;
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[0][m] *= fac1;
    nx3[s] -= nx2[s] * cur4[s];
    nx4[s] -= nx2[s] * cur5[s];
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] -= nx2[s] * rr[0][m];
    const float fac2 = __fdividef(1.0f, nx3[s]);
#pragma unroll
    for (int m = SP_M0(s); m <= SP_M1(s); ++m) rr[1][m] *= fac2;
    tail.cur4[s] = cur4[s];
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) { tail.r2[m] = rr[0][m]; tail.rlast[m] = rr[1][m]; }
}

// Back substitution of the three systems; emit(p, v[5]) receives rows n-2..1.
template <typename Emit>
__device__ __forceinline__ void sp_back_f32(int n, const float* __restrict__ scr, int64_t nlt, int64_t gl,
                                            const SpF32Tail& tail, Emit emit) {
  float b1[5], b2[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const int s = m < 3 ? 0 : m - 2;
    b2[m] = tail.rlast[m];
    b1[m] = tail.r2[m] - tail.cur4[s] * b2[m];
  }
  emit(n - 2, b1);
  for (int p = n - 3; p >= 1; --p) {
    float r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int s = m < 3 ? 0 : m - 2;
      const float l4 = scr[((int64_t)p * 11 + 2 * s) * nlt + gl];
      const float l5 = scr[((int64_t)p * 11 + 2 * s + 1) * nlt + gl];
      r[m] = scr[((int64_t)p * 11 + 6 + m) * nlt + gl] - (l4 * b1[m] + l5 * b2[m]);
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) { b2[m] = b1[m]; b1[m] = r[m]; }
    emit(p, r);
  }
}

// Pass 1 of the mixed SP sweep: all three systems in FP32 from the FP32
// geometry copies; x0 (untransformed) in FP32.  Geometry of point q+1 is
// fetched one row ahead.
template <int DIR>
__global__ void __launch_bounds__(128) k_sp_mixed_solve(Fields F, Consts K, const Work* __restrict__ work,
                                                        float* __restrict__ scr, int64_t nlt,
                                                        float* __restrict__ x0) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  const double* __restrict__ rhs = F.rhs;
  const float* pf = F.primf;
  const int PCV = DIR == 0 ? PS_US : DIR == 1 ? PS_VS : PS_WS;
  // geometry window: values at rows q-1, q, q+1 of the row being assembled
  float gcv[3], grh[3], gsp[3];
  auto geom = [&](int q, float& cv, float& rh, float& sp) {
    const int64_t pt = base + (int64_t)q * st;
    sp_geom_t<DIR, float>(pf[PS_RHOI * NP + pt], pf[PCV * NP + pt], pf[PS_SPEED * NP + pt], K, cv, rh, sp);
  };
  geom(0, gcv[1], grh[1], gsp[1]);
  geom(1, gcv[2], grh[2], gsp[2]);
  gcv[0] = gcv[1]; grh[0] = grh[1]; gsp[0] = gsp[1];
  float ncv = 0.f, nrh = 0.f, nsp = 0.f;
  if (n > 2) geom(2, ncv, nrh, nsp);
  auto row_at = [&](int q, float L[3][5], float r[5]) {
    // window holds q-1, q, q+1 on entry (q+1 from the prefetch)
    sp_assemble<DIR, float, float>(K, q, n, gcv, grh, gsp, L);
    const int64_t pt = base + (int64_t)q * st;
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = (float)rhs[m * NP + pt];
    // shift: q, q+1, prefetched q+2
    gcv[0] = gcv[1]; grh[0] = grh[1]; gsp[0] = gsp[1];
    gcv[1] = gcv[2]; grh[1] = grh[2]; gsp[1] = gsp[2];
    gcv[2] = ncv; grh[2] = nrh; gsp[2] = nsp;
    if (q + 3 <= n - 1) geom(q + 3, ncv, nrh, nsp);
  };
  SpF32Tail tail;
  sp_forward_f32(n, scr, nlt, gl, row_at, tail);
  sp_back_f32(n, scr, nlt, gl, tail, [&](int p, const float v[5]) {
    const int64_t pt = base + (int64_t)p * st;
#pragma unroll
    for (int m = 0; m < 5; ++m) x0[m * NP + pt] = v[m];
  });
}

// Pass 2 of the mixed SP sweep: residual r = b - L x0 of each system in FP64
// (bands of lhsx/lhsy/lhsz assembled in FP64 from a geometry window), the
// FP32 Thomas solve of L d = r, x = x0 + d, the sweep's transform and, after
// the z sweep, add.  x0 is b itself on the boundary rows (identity rows).
template <int DIR>
__global__ void __launch_bounds__(128) k_sp_refine(Fields F, Consts K, const Work* __restrict__ work,
                                                   float* __restrict__ scr, int64_t nlt, int add_u,
                                                   const float* __restrict__ x0f) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int line = w.first + threadIdx.x;
  if (line >= zone_lines(Z, DIR)) return;
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line;
  const int64_t NP = F.NP;
  double* __restrict__ rhs = F.rhs;
  const int PCV = DIR == 0 ? PR_US : DIR == 1 ? PR_VS : PR_WS;
  auto geom = [&](int q, double& cv, double& rh, double& sp) {
    const int64_t pt = base + (int64_t)q * st;
    sp_geom_t<DIR, double>(F.prim[PR_RHOI * NP + pt], F.prim[PCV * NP + pt], F.prim[PR_SPEED * NP + pt], K, cv, rh,
                           sp);
  };
  auto load_x = [&](int q, double x[5]) {
    const int64_t pt = base + (int64_t)q * st;
    if (q < 0 || q > n - 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = 0.0;
    } else if (q == 0 || q == n - 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = rhs[m * NP + pt];
    } else {
#pragma unroll
      for (int m = 0; m < 5; ++m) x[m] = (double)x0f[m * NP + pt];
    }
  };
  // windows for the row being assembled, q: geometry at q-1, q, q+1 and x0 at
  // q-2 .. q+2
  double gcv[3], grh[3], gsp[3], ncv = 0.0, nrh = 0.0, nsp = 0.0;
  double xw[5][5], nxp[5];
  geom(0, gcv[1], grh[1], gsp[1]);
  gcv[0] = gcv[1]; grh[0] = grh[1]; gsp[0] = gsp[1];
  geom(1, gcv[2], grh[2], gsp[2]);
  if (n > 2) geom(2, ncv, nrh, nsp);
  load_x(-2, xw[0]);
  load_x(-1, xw[1]);
  load_x(0, xw[2]);
  load_x(1, xw[3]);
  load_x(2, xw[4]);
  load_x(3, nxp);
  auto row_at = [&](int q, float L[3][5], float r[5]) {
    double Ld[3][5];
    sp_assemble<DIR, double, double>(K, q, n, gcv, grh, gsp, Ld);
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
      for (int b = 0; b < 5; ++b) L[s][b] = (float)Ld[s][b];
    if (q == 0 || q == n - 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) r[m] = 0.f;
    } else {
      const int64_t pt = base + (int64_t)q * st;
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        const int s = m < 3 ? 0 : m - 2;
        const double t = Ld[s][0] * xw[0][m] + Ld[s][1] * xw[1][m] + Ld[s][2] * xw[2][m] + Ld[s][3] * xw[3][m] +
                         Ld[s][4] * xw[4][m];
        r[m] = (float)(rhs[m * NP + pt] - t);
      }
    }
    // advance the windows to row q+1 (values of q+2 / q+3 were fetched one
    // row earlier; fetch the next ones now)
    gcv[0] = gcv[1]; grh[0] = grh[1]; gsp[0] = gsp[1];
    gcv[1] = gcv[2]; grh[1] = grh[2]; gsp[1] = gsp[2];
    gcv[2] = ncv; grh[2] = nrh; gsp[2] = nsp;
    if (q + 3 <= n - 1) geom(q + 3, ncv, nrh, nsp);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int m = 0; m < 5; ++m) xw[k][m] = xw[k + 1][m];
#pragma unroll
    for (int m = 0; m < 5; ++m) xw[4][m] = nxp[m];
    load_x(q + 4, nxp);
  };
  SpF32Tail tail;
  sp_forward_f32(n, scr, nlt, gl, row_at, tail);
  sp_back_f32(n, scr, nlt, gl, tail, [&](int p, const float d[5]) {
    const int64_t pt = base + (int64_t)p * st;
    double v[5], o[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) v[m] = (double)x0f[m * NP + pt] + (double)d[m];
    sp_transform<DIR>(F, K, pt, v, o);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      rhs[m * NP + pt] = o[m];
      if (add_u) F.u[m * NP + pt] += o[m];
    }
  });
}

#if NPBMZ_HAS_FP32
#include "sp_pipelined.cuh"
#include "rhs_df.cuh"
#endif

// ============================================================================
// add (src/BT/add.jl:5-24, src/SP/add.jl:6-26) as a separate phase.
// ============================================================================
__global__ void __launch_bounds__(128) k_add(Fields F, const Work* __restrict__ work) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int q = w.first + threadIdx.x;
  if (q >= Z.nx * Z.ny * Z.nz) return;
  const int i = q % Z.nx, j = (q / Z.nx) % Z.ny, k = q / (Z.nx * Z.ny);
  if (i == 0 || i == Z.nx - 1 || j == 0 || j == Z.ny - 1 || k == 0 || k == Z.nz - 1) return;
  const int64_t p = Z.off + q;
  for (int m = 0; m < 5; ++m) F.u[m * F.NP + p] += F.rhs[m * F.NP + p];
}

#ifndef NPBMZ_NO_LAUNCHERS
// ============================================================================
// host-side launchers (declared in step_launch.h)
// ============================================================================
// Grid of a work-item kernel: one CTA per item, or (persistent) as many CTAs
// as fit on the device at once, each looping over items.
// Grid of a work-list kernel: one CTA per item, or (persist) as many CTAs as
// fit on the SMs looping over the items; ctas_per_sm > 0 makes it persistent
// with at most that many CTAs per SM, which leaves room on every SM for the
// CTAs of kernels running beside it on other streams.
static int item_grid(const void* f, int nwork, int tpb, size_t smem, bool persist, int ctas_per_sm = 0) {
  if (!persist && ctas_per_sm <= 0) return nwork;
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, tpb, smem) != cudaSuccess || per < 1) per = 1;
  if (ctas_per_sm > 0 && ctas_per_sm < per) per = ctas_per_sm;
  return nwork < per * sms ? nwork : per * sms;
}

#if NPBMZ_HAS_FP32
// Blocks of the FP32 x sweeps that read the zone layout: 256 lines per SM at
// once.  A line's points are contiguous there, so a warp's lines lie in 32
// places and each 32-byte sector serves four steps of its line if it stays in
// cache meanwhile; with all the lines that the registers allow (512) it does
// not.  x sweep of 480x320x28, unrefined FP32, by lines per SM: 512 931 us, 384
// 700, 256 535, 192 528 (641 at 384 by the kernel's registers before the scaled
// Jacobians, which left room for more); both passes of the refined sweep
// reading rhs in FP64 1309, 1173, 1153, 1158 (1152 before).
static int x_items(int nwork, int tpb) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::min(nwork, std::max(1, 256 / tpb) * sms);
}
#endif

void launch_prim_w(bool sp, const Fields& F, const Consts& K, const Work* work, int nwork, cudaStream_t s,
                   bool persist) {
  if (nwork <= 0) return;
  if (sp) k_prim_w<true><<<item_grid((const void*)k_prim_w<true>, nwork, 128, 0, persist), 128, 0, s>>>(F, K, work, nwork);
  else k_prim_w<false><<<item_grid((const void*)k_prim_w<false>, nwork, 128, 0, persist), 128, 0, s>>>(F, K, work, nwork);
}

void launch_prim(bool sp, const Fields& F, const Consts& K, int64_t lo, int64_t hi, cudaStream_t s) {
  if (hi <= lo) return;
  int64_t g = (hi - lo + 255) / 256;
  const int grid = (int)(g > 8192 ? 8192 : g);
  if (sp) k_prim<true><<<grid, 256, 0, s>>>(F, K, lo, hi);
  else k_prim<false><<<grid, 256, 0, s>>>(F, K, lo, hi);
}

void launch_rhs(bool tx, bool norm, const Fields& F, const Consts& K, const Work* work, int nwork, double* partials,
                cudaStream_t s, const RhsF64Consts* rc, bool persist) {
  if (nwork <= 0) return;
#if NPBMZ_HAS_FP32
  if (F.flux && F.fdt && rc) {
#define NPBMZ_RHS_FLUX(A, B)                                                                                  \
  k_rhs_flux<A, B><<<item_grid((const void*)k_rhs_flux<A, B>, nwork, 128, 0, persist), 128, 0, s>>>(F, K, *rc, work, \
                                                                                                  nwork, partials)
    if (tx) {
      if (norm) NPBMZ_RHS_FLUX(true, true);
      else NPBMZ_RHS_FLUX(true, false);
    } else {
      if (norm) NPBMZ_RHS_FLUX(false, true);
      else NPBMZ_RHS_FLUX(false, false);
    }
#undef NPBMZ_RHS_FLUX
    return;
  }
#endif
  if (tx) {
    if (norm) k_rhs<true, true><<<nwork, 128, 0, s>>>(F, K, work, partials);
    else k_rhs<true, false><<<nwork, 128, 0, s>>>(F, K, work, partials);
  } else {
    if (norm) k_rhs<false, true><<<nwork, 128, 0, s>>>(F, K, work, partials);
    else k_rhs<false, false><<<nwork, 128, 0, s>>>(F, K, work, partials);
  }
}

template <typename T>
static void launch_solve_t(bool sp, int dir, const Fields& F, const Consts& K, const Work* work, int nwork, int tpb,
                           void* scratch, int64_t nlt, int add_u, double* out, int transform, cudaStream_t s) {
  T* scr = reinterpret_cast<T*>(scratch);
  if (sp) {
    if (dir == 0) k_sp_solve<0, T><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, out, transform);
    else if (dir == 1) k_sp_solve<1, T><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, out, transform);
    else k_sp_solve<2, T><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, out, transform);
  } else {
#if NPBMZ_HAS_FP32
    const int gx = sizeof(T) == sizeof(float) ? x_items(nwork, tpb) : nwork;
    if (dir == 0) k_bt_line<0, T><<<gx, tpb, 0, s>>>(F, K, work, nwork, scr, nlt, add_u);
    else if (dir == 1) k_bt_line<1, T><<<nwork, tpb, 0, s>>>(F, K, work, nwork, scr, nlt, add_u);
    else k_bt_line<2, T><<<nwork, tpb, 0, s>>>(F, K, work, nwork, scr, nlt, add_u);
#else
    if (dir == 0) k_bt_solve<0><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u);
    else if (dir == 1) k_bt_solve<1><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u);
    else k_bt_solve<2><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u);
#endif
  }
}

// mode 4: one fused refined FP32 step (6: BT, two threads per line); mode 0:
// FP64 in place (5: BT, twelve lanes per line); 1: FP32 in place; 2: FP32 + refinement with a
// double-float residual (BT; SP: FP64 residual); 3: FP32 + refinement with
// an FP64 residual (xw: a [5][NP] buffer for the first solution).
void launch_solve(bool sp, int mode, int dir, const Fields& F, const Consts& K, const Work* work, int nwork, int tpb,
                  void* scratch, int64_t nlt, int add_u, double* xw, cudaStream_t s, bool persist, int ctas_per_sm) {
  if (nwork <= 0) return;
#if NPBMZ_HAS_FP32
  if (mode == 1) { launch_solve_t<float>(sp, dir, F, K, work, nwork, tpb, scratch, nlt, add_u, F.rhs, 1, s); return; }
  if (mode == 4 && sp) {
    // one fused step, SP: the pipelined passes with a double-float residual;
    // x and y hand their transformed results on as double-float
    float* scr = reinterpret_cast<float*>(scratch);
    float* x0 = reinterpret_cast<float*>(xw);
    const size_t sm_m = pls_mixed_smem(tpb), sm_r = pls_refine_smem(tpb, dir != 2);
#define NPBMZ_SPL(D, OD)                                                                                          \
  do {                                                                                                            \
    k_sp_mixed_pl<D><<<item_grid((const void*)k_sp_mixed_pl<D>, nwork, tpb, sm_m, persist, ctas_per_sm), tpb,     \
                       sm_m, s>>>(                                                                                \
        F, K, work, nwork, scr, nlt, x0);                                                                         \
    k_sp_refine_pl<D, OD><<<item_grid((const void*)k_sp_refine_pl<D, OD>, nwork, tpb, sm_r, persist, ctas_per_sm), \
                            tpb, sm_r,                                                                            \
                            s>>>(F, K, work, nwork, scr, nlt, add_u, x0);                                         \
  } while (0)
    if (dir == 0) {
      NPBMZ_SPL(0, true);
      k_xline_back<<<nwork, 256, 0, s>>>(F, work, nwork, tpb);
    } else if (dir == 1) NPBMZ_SPL(1, true);
    else NPBMZ_SPL(2, false);
#undef NPBMZ_SPL
    return;
  }
  if ((mode == 4 || mode == 6) && !sp) {
    // one fused step: b of the x sweep comes from compute_rhs's double-float
    // copy, x and y hand their results on as double-float (x through its
    // x-line-major copy), z writes FP64 rhs (and u)
    float* scr = reinterpret_cast<float*>(scratch);
    float* x0 = reinterpret_cast<float*>(xw);
    const bool two = mode == 6;
    const int thr = two ? 2 * tpb : tpb;
    const size_t sm_m = pl_mixed_smem(tpb, two), sm_r = pl_refine_smem(tpb, two);
#define NPBMZ_PL(D, OD, TW)                                                                                          \
  do {                                                                                                               \
    k_bt_mixed_pl<D, TW><<<item_grid((const void*)k_bt_mixed_pl<D, TW>, nwork, thr, sm_m, persist, ctas_per_sm), thr, \
                           sm_m, s>>>(F, K, work, nwork, scr, nlt, x0);                                              \
    k_bt_refine_pl<D, OD, TW><<<item_grid((const void*)k_bt_refine_pl<D, OD, TW>, nwork, thr, sm_r, persist,         \
                                          ctas_per_sm),                                                              \
                                thr, sm_r, s>>>(F, K, work, nwork, scr, nlt, add_u, x0);                             \
  } while (0)
    if (dir == 0) {
      if (two) NPBMZ_PL(0, true, true);
      else NPBMZ_PL(0, true, false);
      k_xline_back<<<nwork, 256, 0, s>>>(F, work, nwork, tpb);
    } else if (dir == 1) {
      if (two) NPBMZ_PL(1, true, true);
      else NPBMZ_PL(1, true, false);
    } else {
      if (two) NPBMZ_PL(2, false, true);
      else NPBMZ_PL(2, false, false);
    }
#undef NPBMZ_PL
    return;
  }
  if (mode == 2 || mode == 3) {
    const bool resid64 = mode == 3;
    float* scr = reinterpret_cast<float*>(scratch);
    if (sp) {
      float* x0 = reinterpret_cast<float*>(xw);
      if (dir == 0) {
        k_sp_mixed_solve<0><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, x0);
        k_sp_refine<0><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      } else if (dir == 1) {
        k_sp_mixed_solve<1><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, x0);
        k_sp_refine<1><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      } else {
        k_sp_mixed_solve<2><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, x0);
        k_sp_refine<2><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      }
    } else {
      float* x0 = reinterpret_cast<float*>(xw);
      if (dir == 0) {
        k_bt_mixed_solve<0><<<x_items(nwork, tpb), tpb, 0, s>>>(F, K, work, nwork, scr, nlt, x0);
        if (resid64) k_bt_refine<0><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
        else k_bt_refine_df<0><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      } else if (dir == 1) {
        k_bt_mixed_solve<1><<<nwork, tpb, 0, s>>>(F, K, work, nwork, scr, nlt, x0);
        if (resid64) k_bt_refine<1><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
        else k_bt_refine_df<1><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      } else {
        k_bt_mixed_solve<2><<<nwork, tpb, 0, s>>>(F, K, work, nwork, scr, nlt, x0);
        if (resid64) k_bt_refine<2><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
        else k_bt_refine_df<2><<<nwork, tpb, 0, s>>>(F, K, work, scr, nlt, add_u, x0);
      }
    }
    return;
  }
#else
  (void)xw;
#endif
#if NPBMZ_HAS_FP32
  if (mode == 5) {
    const dim3 grid(nwork, (tpb + BTS_LINES - 1) / BTS_LINES);
    double* scr = reinterpret_cast<double*>(scratch);
    if (dir == 0) k_bt_line12<0><<<grid, 64, BTS_SMEM, s>>>(F, K, work, tpb, scr, nlt, add_u);
    else if (dir == 1) k_bt_line12<1><<<grid, 64, BTS_SMEM, s>>>(F, K, work, tpb, scr, nlt, add_u);
    else k_bt_line12<2><<<grid, 64, BTS_SMEM, s>>>(F, K, work, tpb, scr, nlt, add_u);
    return;
  }
#endif
  (void)mode;
  launch_solve_t<double>(sp, dir, F, K, work, nwork, tpb, scratch, nlt, add_u, F.rhs, 1, s);
}

#if NPBMZ_HAS_FP32
// Opt the pipelined sweeps into their dynamic shared memory (above 48 KB for
// 128 threads per CTA); called once per handle, outside any stream capture.
int configure_kernels() {
  size_t cap_b = pl_refine_smem(128, true);
  for (size_t b : {pl_mixed_smem(128, true), pls_mixed_smem(128), pls_refine_smem(128, false)})
    if (b > cap_b) cap_b = b;
  const int cap = (int)cap_b;
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f) {
    const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
    if (r != cudaSuccess) e = r;
  };
  set((const void*)k_bt_mixed_pl<0, false>);
  set((const void*)k_bt_mixed_pl<0, true>);
  set((const void*)k_bt_mixed_pl<1, false>);
  set((const void*)k_bt_mixed_pl<1, true>);
  set((const void*)k_bt_mixed_pl<2, false>);
  set((const void*)k_bt_mixed_pl<2, true>);
  set((const void*)k_bt_refine_pl<0, true, false>);
  set((const void*)k_bt_refine_pl<0, true, true>);
  set((const void*)k_bt_refine_pl<1, true, false>);
  set((const void*)k_bt_refine_pl<1, true, true>);
  set((const void*)k_bt_refine_pl<2, false, false>);
  set((const void*)k_bt_refine_pl<2, false, true>);
  set((const void*)k_sp_mixed_pl<0>);
  set((const void*)k_sp_mixed_pl<1>);
  set((const void*)k_sp_mixed_pl<2>);
  set((const void*)k_sp_refine_pl<0, true>);
  set((const void*)k_sp_refine_pl<1, true>);
  set((const void*)k_sp_refine_pl<2, false>);
  return e == cudaSuccess ? 0 : -1;
}

void launch_xline_ends(const Fields& F, const Work* work, int nwork, int tpb, cudaStream_t s) {
  if (nwork > 0) k_xline_ends<<<nwork, tpb, 0, s>>>(F, work);
}

void launch_prim_df(bool sp, const Fields& F, const RhsDfConsts& C, const Work* work, int nwork, cudaStream_t s,
                    bool persist) {
  if (nwork <= 0) return;
  if (sp) k_prim_df<true><<<item_grid((const void*)k_prim_df<true>, nwork, 128, 0, persist), 128, 0, s>>>(F, C, work, nwork);
  else k_prim_df<false><<<item_grid((const void*)k_prim_df<false>, nwork, 128, 0, persist), 128, 0, s>>>(F, C, work, nwork);
}

void launch_rhs_df(bool tx, bool norm, const Fields& F, const RhsDfConsts& C, const Work* work, int nwork,
                   double* partials, cudaStream_t s, bool persist) {
  if (nwork <= 0) return;
#define NPBMZ_RHS_DF(A, B)                                                                                      \
  do {                                                                                                          \
    if (C.exact_w)                                                                                              \
      k_rhs_df<A, B, true><<<item_grid((const void*)k_rhs_df<A, B, true>, nwork, 128, 0, persist), 128, 0, s>>>(  \
          F, C, work, nwork, partials);                                                                         \
    else                                                                                                        \
      k_rhs_df<A, B, false><<<item_grid((const void*)k_rhs_df<A, B, false>, nwork, 128, 0, persist), 128, 0, s>>>( \
          F, C, work, nwork, partials);                                                                         \
  } while (0)
  if (tx) {
    if (norm) NPBMZ_RHS_DF(true, true);
    else NPBMZ_RHS_DF(true, false);
  } else {
    if (norm) NPBMZ_RHS_DF(false, true);
    else NPBMZ_RHS_DF(false, false);
  }
#undef NPBMZ_RHS_DF
}

void launch_xline_copy(bool sp, const Fields& F, const Work* work, int nwork, int lpi, cudaStream_t s) {
  if (nwork <= 0) return;
  if (sp) k_xline_copy<true><<<nwork, 256, 0, s>>>(F, work, nwork, lpi);
  else k_xline_copy<false><<<nwork, 256, 0, s>>>(F, work, nwork, lpi);
}

void launch_rhs_xc(bool tx, bool norm, const Fields& F, const Consts& K, const RhsF64Consts& rc, const Work* work,
                   int nwork, double* partials, const Work* cwork, int ncopy, int lpi, cudaStream_t s, bool persist) {
  if (nwork + ncopy <= 0) return;
#define NPBMZ_RHS_XC(A, B)                                                                                   \
  k_rhs_flux_xc<A, B><<<item_grid((const void*)k_rhs_flux_xc<A, B>, nwork + ncopy, 128, 0, persist), 128, 0, s>>>( \
      F, K, rc, work, nwork, partials, cwork, ncopy, lpi)
  if (tx) {
    if (norm) NPBMZ_RHS_XC(true, true);
    else NPBMZ_RHS_XC(true, false);
  } else {
    if (norm) NPBMZ_RHS_XC(false, true);
    else NPBMZ_RHS_XC(false, false);
  }
#undef NPBMZ_RHS_XC
}

void launch_scale(const double* src, double* dst, double a, int64_t n, cudaStream_t s) {
  int64_t g = (n + 255) / 256;
  k_scale<<<(int)(g > 8192 ? 8192 : g), 256, 0, s>>>(src, dst, a, n);
}

void launch_split_f2(const double* src, float2* dst, int64_t NP, cudaStream_t s) {
  int64_t g = (5 * NP + 255) / 256;
  k_split_f2<<<(int)(g > 8192 ? 8192 : g), 256, 0, s>>>(src, dst, NP);
}

void launch_split_df(const double* src, float* dst, int64_t NP, cudaStream_t s) {
  int64_t g = (5 * NP + 255) / 256;
  k_split_df<<<(int)(g > 8192 ? 8192 : g), 256, 0, s>>>(src, dst, NP);
}
#endif

void launch_add(const Fields& F, const Work* work, int nwork, cudaStream_t s) {
  if (nwork > 0) k_add<<<nwork, 128, 0, s>>>(F, work);
}

#endif  // NPBMZ_NO_LAUNCHERS

}  // namespace NPBMZ_NS
}  // namespace npbmz
