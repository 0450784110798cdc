// lu_kernels.cuh -- the LU-MZ device code (NPBApps.jl src/LU), compiled
// twice into namespaces named by LU_NS: lu_exact.cu with -fmad=false (every
// FP64 statement rounds as the reference's Julia does, bit-for-bit the
// oracle) and lu_fast.cu with -fmad=true (a*b+c contracted to FMA).
#pragma once
#ifndef LU_NS
#error "define LU_NS before including lu_kernels.cuh"
#endif
#include "lu_types.h"

namespace npbmz_lu {
namespace LU_NS {

// ---- exact solution (src/LU/exact.jl) ---------------------------------------
__device__ inline void exact_point(const CeTable& ce, int i, int j, int k, int nx0, int ny0, int nz0, double out[5]) {
  const double xi = (double)(i - 1) / (nx0 - 1);
  const double eta = (double)(j - 1) / (ny0 - 1);
  const double zeta = (double)(k - 1) / (nz0 - 1);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const double* c = ce.c[m];
    out[m] = c[0] + (c[1] + (c[4] + (c[7] + c[10] * xi) * xi) * xi) * xi +
             (c[2] + (c[5] + (c[8] + c[11] * eta) * eta) * eta) * eta +
             (c[3] + (c[6] + (c[9] + c[12] * zeta) * zeta) * zeta) * zeta;
  }
}

// ---- rhs / erhs point operator (src/LU/rhs.jl, src/LU/erhs.jl) -------------
// o: the point's output, holding -frct (rhs) or 0 (erhs) on entry.  ERHS
// selects erhs's z second difference order (g(k+1) first) and its viscous
// association ((o + A) + B instead of o + (A + B)).
template <bool ERHS>
__device__ inline double visc_up(double o, double a, double b) {
  return ERHS ? (o + a) + b : o + (a + b);
}

// The flux quantities of one point; returns q.
__device__ __forceinline__ double prim_point(const double g[5], double pr[PR_COUNT]) {
  const double tmp = 1.0e+00 / g[0];
  pr[PR_RHO] = tmp;
  pr[PR_U21] = tmp * g[1];
  pr[PR_U31] = tmp * g[2];
  pr[PR_U41] = tmp * g[3];
  pr[PR_U51] = tmp * g[4];
  pr[PR_S] = pr[PR_U21] * pr[PR_U21] + pr[PR_U31] * pr[PR_U31] + pr[PR_U41] * pr[PR_U41];
  const double u21 = div_y(g[1], g[0], tmp), u31 = div_y(g[2], g[0], tmp), u41 = div_y(g[3], g[0], tmp);
  const double q = div_y(0.50e+00 * (g[1] * g[1] + g[2] * g[2] + g[3] * g[3]), g[0], tmp);
  const double pres = c2 * (g[4] - q), h = c1 * g[4] - c2 * q;
  const double vel[3] = {u21, u31, u41};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double f = g[m + 1] * vel[d];
      pr[PR_F + 4 * d + m] = m == d ? f + pres : f;
    }
    pr[PR_F + 4 * d + 3] = h * vel[d];
  }
  return q;
}

__device__ __forceinline__ void store_prim(double* prim, long long NP, long long p, const double g[5]) {
  double pr[PR_COUNT];
  prim_point(g, pr);
#pragma unroll
  for (int q = 0; q < PR_COUNT; ++q) prim[q * NP + p] = pr[q];
}

// Products with 2, 4 and dssp = 1/4 are exact, so fma rounds them and the sum
// once, as the separate operations do: the second differences and the
// fourth-difference dissipation take an FP64 instruction less for each.
static_assert(dssp == 0.25, "the dissipation's fma needs a power of two");

// o - dssp times the fourth difference of u at position q (1-based, 2..n-1) of
// an axis of n >= 6 points: the reference's start, middle and end stencils are
// the middle one, whose missing terms enter as zeros (x - 0 and 0 + x are x),
// with 5 instead of 6 at the centre of the outermost two; no lane diverges.
__device__ __forceinline__ double dissip(double o, int q, int n, double um2, double um1, double u0, double up1,
                                         double up2) {
  const double a = q >= 4 ? um2 : 0.0, b = q >= 3 ? um1 : 0.0, d = q <= n - 2 ? up1 : 0.0, e = q <= n - 3 ? up2 : 0.0;
  const double w = q == 2 || q == n - 1 ? 5.0e+00 : 6.0e+00;
  return fma(-dssp, fma(-4.0e+00, d, fma(-4.0e+00, b, a) + w * u0) + e, o);
}
// The same on an axis of 5 points, where two stencils apply at the middle one.
__device__ __noinline__ double dissip5(double o, int q, double um2, double um1, double u0, double up1, double up2) {
  if (q == 2) o = o - dssp * (+5.0e+00 * u0 - 4.0e+00 * up1 + up2);
  if (q == 3) o = o - dssp * (-4.0e+00 * um1 + 6.0e+00 * u0 - 4.0e+00 * up1 + up2);
  if (q == 3) o = o - dssp * (um2 - 4.0e+00 * um1 + 6.0e+00 * u0 - 4.0e+00 * up1);
  if (q == 4) o = o - dssp * (um2 - 4.0e+00 * um1 + 5.0e+00 * u0);
  return o;
}

// One direction of the operator at point p (position q of an axis of n points,
// stride st): the reference's statements, in their order.
template <bool ERHS, int D>
__device__ __forceinline__ void flux_dir(const double* __restrict__ g, const double* __restrict__ prim, long long NP,
                                         long long p, long long st, int q, int n, double t1, double t2, double t3,
                                         double d1, double o[5]) {
  const long long a = p + st, b = p - st;
  // convective flux
  o[0] = o[0] - t2 * (g[(D + 1) * NP + a] - g[(D + 1) * NP + b]);
#pragma unroll
  for (int m = 1; m < 5; ++m) {
    const double* f = prim + (PR_F + 4 * D + m - 1) * NP;
    o[m] = o[m] - t2 * (f[a] - f[b]);
  }
  // viscous fluxes between the point and its neighbours
  auto visc = [&](long long hi, long long lo, double f[5]) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
      f[m + 1] = (D == m ? (4.0e+00 / 3.0e+00) * t3 : t3) * (prim[(PR_U21 + m) * NP + hi] - prim[(PR_U21 + m) * NP + lo]);
    const double ui = prim[(PR_U21 + D) * NP + hi], um = prim[(PR_U21 + D) * NP + lo];
    f[4] = 0.50e+00 * (1.0e+00 - c1 * c5) * t3 * (prim[PR_S * NP + hi] - prim[PR_S * NP + lo]) +
           (1.0e+00 / 6.0e+00) * t3 * (ui * ui - um * um) +
           c1 * c5 * t3 * (prim[PR_U51 * NP + hi] - prim[PR_U51 * NP + lo]);
  };
  double fp[5], fm[5];
  visc(a, p, fp);
  visc(p, b, fm);
  // second difference: x and y take g(-1) first; z too in rhs, g(+1) in erhs
  auto second = [&](int m) {
    const double* u = g + m * NP;
    const double x = D == 2 && ERHS ? u[a] : u[b], y = D == 2 && ERHS ? u[b] : u[a];
    return fma(-2.0e+00, u[p], x) + y;
  };
  o[0] = o[0] + d1 * t1 * second(0);
#pragma unroll
  for (int m = 1; m < 5; ++m) o[m] = visc_up<ERHS>(o[m], t3 * c3 * c4 * (fp[m] - fm[m]), d1 * t1 * second(m));
  const long long p2 = q <= n - 2 ? a + st : p, m2 = q >= 3 ? b - st : p;
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const double* u = g + m * NP;
    o[m] = n == 5 ? dissip5(o[m], q, u[m2], u[b], u[p], u[a], u[p2]) : dissip(o[m], q, n, u[m2], u[b], u[p], u[a], u[p2]);
  }
}

template <bool ERHS>
__device__ __forceinline__ void flux_point(const double* __restrict__ g, const double* __restrict__ prim, long long NP,
                                           const LuZone& Z, int i, int j, int k, double o[5]) {
  static_assert(dx1 == dx5 && dy1 == dy5 && dz1 == dz5, "one factor per direction");
  const long long p = pidx(Z, i, j, k);
  flux_dir<ERHS, 0>(g, prim, NP, p, 1, i, Z.nx, Z.tx1, Z.tx2, Z.tx3, dx1, o);
  flux_dir<ERHS, 1>(g, prim, NP, p, Z.nx, j, Z.ny, Z.ty1, Z.ty2, Z.ty3, dy1, o);
  flux_dir<ERHS, 2>(g, prim, NP, p, (long long)Z.nx * Z.ny, k, Z.nz, Z.tz1, Z.tz2, Z.tz3, dz1, o);
}

__device__ inline bool decode(const LuZone& Z, int q, int& i, int& j, int& k) {
  if (q >= Z.np) return false;
  i = q % Z.nx + 1;
  j = (q / Z.nx) % Z.ny + 1;
  k = q / (Z.nx * Z.ny) + 1;
  return true;
}

__device__ inline bool interior(const LuZone& Z, int i, int j, int k) {
  return i >= 2 && i <= Z.nx - 1 && j >= 2 && j <= Z.ny - 1 && k >= 2 && k <= Z.nz - 1;
}

// Bound by the FP64 pipe: 309 FP64 instructions a point without
// contraction (444 with the convective fluxes formed at every neighbour, the
// products with 2, 4 and 1/4 apart, and a divergent branch per stencil).
// 480x320x28: 5.00 -> 2.58 ms; contracted 3.2 -> 1.98 ms.
// rhs (ERHS = false: g = u, out = rsd starting at -frct) or erhs's flux part
// (ERHS = true: g = the exact polynomial in rsd, out = frct starting at 0)
template <bool ERHS>
__global__ void __launch_bounds__(TPB) k_lu_rhs(LuDev D, const LuWork* __restrict__ work, const double* g,
                                                const double* __restrict__ prim, double* out) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  int i, j, k;
  if (!decode(Z, w.first + threadIdx.x, i, j, k)) return;
  const long long p = pidx(Z, i, j, k);
  double o[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) o[m] = ERHS ? 0.0 : -D.frct[m * D.NP + p];
  if (interior(Z, i, j, k)) flux_point<ERHS>(g, prim, D.NP, Z, i, j, k, o);
#pragma unroll
  for (int m = 0; m < 5; ++m) out[m * D.NP + p] = o[m];
}

// setbv + setiv (src/LU/setbv.jl, src/LU/setiv.jl); every face point of
// setbv gets exact() of its own (i, j, k), whichever face writes it last
__global__ void __launch_bounds__(TPB) k_lu_init(LuDev D, const LuWork* __restrict__ work, CeTable ce) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  int i, j, k;
  if (!decode(Z, w.first + threadIdx.x, i, j, k)) return;
  const int nx = Z.nx, ny = Z.ny, nz = Z.nz;
  const long long p = pidx(Z, i, j, k);
  double out[5];
  if (!interior(Z, i, j, k)) {
    exact_point(ce, i, j, k, nx, ny, nz, out);
  } else {
    const double zeta = (double)(k - 1) / (nz - 1);
    const double eta = (double)(j - 1) / (ny - 1);
    const double xi = (double)(i - 1) / (nx - 1);
    double a1[5], a2[5], b1[5], b2[5], g1[5], g2[5];
    exact_point(ce, 1, j, k, nx, ny, nz, a1);
    exact_point(ce, nx, j, k, nx, ny, nz, a2);
    exact_point(ce, i, 1, k, nx, ny, nz, b1);
    exact_point(ce, i, ny, k, nx, ny, nz, b2);
    exact_point(ce, i, j, 1, nx, ny, nz, g1);
    exact_point(ce, i, j, nz, nx, ny, nz, g2);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double pxi = (1.0e+00 - xi) * a1[m] + xi * a2[m];
      const double peta = (1.0e+00 - eta) * b1[m] + eta * b2[m];
      const double pzeta = (1.0e+00 - zeta) * g1[m] + zeta * g2[m];
      out[m] = pxi + peta + pzeta - pxi * peta - peta * pzeta - pzeta * pxi + pxi * peta * pzeta;
    }
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) D.u[m * D.NP + p] = out[m];
}

// erhs's first part: rsd = the exact polynomial (non-Horner, src/LU/erhs.jl:24-47)
__global__ void __launch_bounds__(TPB) k_lu_poly(LuDev D, const LuWork* __restrict__ work, CeTable ce) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  int i, j, k;
  if (!decode(Z, w.first + threadIdx.x, i, j, k)) return;
  const long long p = pidx(Z, i, j, k);
  const double zeta = (double)(k - 1) / (Z.nz - 1);
  const double eta = (double)(j - 1) / (Z.ny - 1);
  const double xi = (double)(i - 1) / (Z.nx - 1);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const double* c = ce.c[m];
    D.rsd[m * D.NP + p] = c[0] + c[1] * xi + c[2] * eta + c[3] * zeta + c[4] * xi * xi + c[5] * eta * eta +
                          c[6] * zeta * zeta + c[7] * xi * xi * xi + c[8] * eta * eta * eta +
                          c[9] * zeta * zeta * zeta + c[10] * xi * xi * xi * xi + c[11] * eta * eta * eta * eta +
                          c[12] * zeta * zeta * zeta * zeta;
  }
}

// rsd *= dt (SCALE) or u += tmp * rsd (UPDATE, with the point's prim
// planes refreshed from the new u) on the interior
template <bool UPDATE>
__global__ void __launch_bounds__(TPB) k_lu_pointwise(LuDev D, const LuWork* __restrict__ work, double tmp) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  int i, j, k;
  if (!decode(Z, w.first + threadIdx.x, i, j, k) || !interior(Z, i, j, k)) return;
  const long long p = pidx(Z, i, j, k);
  if (UPDATE) {
    double g[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      g[m] = D.u[m * D.NP + p] + tmp * D.rsd[m * D.NP + p];
      D.u[m * D.NP + p] = g[m];
    }
    double pr[PR_COUNT];
    const double qk = prim_point(g, pr);
#pragma unroll
    for (int q = 0; q < PR_COUNT; ++q) D.prim[q * D.NP + p] = pr[q];
    if (D.health) {
      // on the bit patterns (integer pipe): positive and finite
      const double pres = g[4] - qk;
      const unsigned long long br = (unsigned long long)__double_as_longlong(g[0]);
      const unsigned long long bp = (unsigned long long)__double_as_longlong(pres);
      const bool rho_ok = br - 1ull < 0x7FEFFFFFFFFFFFFFull, p_ok = bp - 1ull < 0x7FEFFFFFFFFFFFFFull;
      if (!(rho_ok && p_ok)) {
        const bool p_finite = (bp & 0x7FF0000000000000ull) != 0x7FF0000000000000ull;
        const unsigned bits = (rho_ok ? 0u : LU_STATE_DENSITY) |
                              (p_ok ? 0u : p_finite ? LU_STATE_PRESSURE : LU_STATE_NONFINITE);
        atomicOr(D.health, (unsigned long long)bits);
        atomicMin(D.health + 1, (unsigned long long)p);
      }
    }
  } else {
#pragma unroll
    for (int m = 0; m < 5; ++m) D.rsd[m * D.NP + p] = D.dt * D.rsd[m * D.NP + p];
  }
}

// prim planes of g (u, or erhs's exact polynomial) at every point
__global__ void __launch_bounds__(TPB) k_lu_prim(LuDev D, const LuWork* __restrict__ work, const double* g) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  const int q = w.first + threadIdx.x;
  if (q >= Z.np) return;
  const long long p = Z.off + q;
  double v[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) v[m] = g[m * D.NP + p];
  store_prim(D.prim, D.NP, p, v);
}

// ---- Jacobian blocks of jacld / jacu (src/LU/jacld.jl, src/LU/jacu.jl) -----
// the diagonal block (identical in jacld and jacu) at the point's own state
__device__ __forceinline__ void jac_d(const JC& J, double r1, double u2, double u3, double u4, double u5,
                                      double d[5][5]) {
  const double dt = J.dt, tx1 = J.tx1, ty1 = J.ty1, tz1 = J.tz1;
  const double tmp1 = r1, tmp2 = tmp1 * tmp1, tmp3 = tmp1 * tmp2;
  d[0][0] = 1.0e+00 + dt * 2.0e+00 * (tx1 * dx1 + ty1 * dy1 + tz1 * dz1);
  d[0][1] = 0.0; d[0][2] = 0.0; d[0][3] = 0.0; d[0][4] = 0.0;
  d[1][0] = dt * 2.0e+00 * (tx1 * (-r43 * c34 * tmp2 * u2) + ty1 * (-c34 * tmp2 * u2) + tz1 * (-c34 * tmp2 * u2));
  d[1][1] = 1.0e+00 + dt * 2.0e+00 * (tx1 * r43 * c34 * tmp1 + ty1 * c34 * tmp1 + tz1 * c34 * tmp1) +
            dt * 2.0e+00 * (tx1 * dx2 + ty1 * dy2 + tz1 * dz2);
  d[1][2] = 0.0; d[1][3] = 0.0; d[1][4] = 0.0;
  d[2][0] = dt * 2.0e+00 * (tx1 * (-c34 * tmp2 * u3) + ty1 * (-r43 * c34 * tmp2 * u3) + tz1 * (-c34 * tmp2 * u3));
  d[2][1] = 0.0;
  d[2][2] = 1.0e+00 + dt * 2.0e+00 * (tx1 * c34 * tmp1 + ty1 * r43 * c34 * tmp1 + tz1 * c34 * tmp1) +
            dt * 2.0e+00 * (tx1 * dx3 + ty1 * dy3 + tz1 * dz3);
  d[2][3] = 0.0; d[2][4] = 0.0;
  d[3][0] = dt * 2.0e+00 * (tx1 * (-c34 * tmp2 * u4) + ty1 * (-c34 * tmp2 * u4) + tz1 * (-r43 * c34 * tmp2 * u4));
  d[3][1] = 0.0; d[3][2] = 0.0;
  d[3][3] = 1.0e+00 + dt * 2.0e+00 * (tx1 * c34 * tmp1 + ty1 * c34 * tmp1 + tz1 * r43 * c34 * tmp1) +
            dt * 2.0e+00 * (tx1 * dx4 + ty1 * dy4 + tz1 * dz4);
  d[3][4] = 0.0;
  d[4][0] = dt * 2.0e+00 *
            (tx1 * (-(r43 * c34 - c1345) * tmp3 * (u2 * u2) - (c34 - c1345) * tmp3 * (u3 * u3) -
                    (c34 - c1345) * tmp3 * (u4 * u4) - (c1345)*tmp2 * u5) +
             ty1 * (-(c34 - c1345) * tmp3 * (u2 * u2) - (r43 * c34 - c1345) * tmp3 * (u3 * u3) -
                    (c34 - c1345) * tmp3 * (u4 * u4) - (c1345)*tmp2 * u5) +
             tz1 * (-(c34 - c1345) * tmp3 * (u2 * u2) - (c34 - c1345) * tmp3 * (u3 * u3) -
                    (r43 * c34 - c1345) * tmp3 * (u4 * u4) - (c1345)*tmp2 * u5));
  d[4][1] = dt * 2.0e+00 *
            (tx1 * (r43 * c34 - c1345) * tmp2 * u2 + ty1 * (c34 - c1345) * tmp2 * u2 + tz1 * (c34 - c1345) * tmp2 * u2);
  d[4][2] = dt * 2.0e+00 *
            (tx1 * (c34 - c1345) * tmp2 * u3 + ty1 * (r43 * c34 - c1345) * tmp2 * u3 + tz1 * (c34 - c1345) * tmp2 * u3);
  d[4][3] = dt * 2.0e+00 *
            (tx1 * (c34 - c1345) * tmp2 * u4 + ty1 * (c34 - c1345) * tmp2 * u4 + tz1 * (r43 * c34 - c1345) * tmp2 * u4);
  d[4][4] = 1.0e+00 + dt * 2.0e+00 * (tx1 * c1345 * tmp1 + ty1 * c1345 * tmp1 + tz1 * c1345 * tmp1) +
            dt * 2.0e+00 * (tx1 * dx5 + ty1 * dy5 + tz1 * dz5);
}

// The state-dependent entries of jacld's (lo: the block the point at +1 in DIR
// reads) and jacu's (up: the point at -1) off-diagonal blocks of direction
// DIR (0 x, 1 y, 2 z) from one point's state; r1 = 1/u1 (the reference's tmp1:
// the PR_RHO plane).  The entries are the reference's statements; jacld's
// differ from jacu's in the sign of the convective term, their first, alone,
// so each term is formed once and the two entries are its sums: about 95 FP64
// operations a direction.
template <int DIR>
__device__ __forceinline__ void jac_off(const JC& J, double r1, double u2, double u3, double u4, double u5,
                                        double lo[5][5], double up[5][5]) {
  const double dt = J.dt;
  const double tmp1 = r1, tmp2 = tmp1 * tmp1, tmp3 = tmp1 * tmp2;
#define NPBMZ_LU_OFF(r, c, P, rest) \
  {                                 \
    const double conv = P;          \
    lo[r][c] = -conv rest;          \
    up[r][c] = conv rest;           \
  }
  if (DIR == 2) {
    const double tz1 = J.tz1, tz2 = J.tz2;
    NPBMZ_LU_OFF(1, 0, (dt * tz2 * (-(u2 * u4) * tmp2)), - dt * tz1 * (-c34 * tmp2 * u2))
    NPBMZ_LU_OFF(1, 1, (dt * tz2 * (u4 * tmp1)), - dt * tz1 * c34 * tmp1 - dt * tz1 * dz2)
    NPBMZ_LU_OFF(1, 3, (dt * tz2 * (u2 * tmp1)), )
    NPBMZ_LU_OFF(2, 0, (dt * tz2 * (-(u3 * u4) * tmp2)), - dt * tz1 * (-c34 * tmp2 * u3))
    NPBMZ_LU_OFF(2, 2, (dt * tz2 * (u4 * tmp1)), - dt * tz1 * (c34 * tmp1) - dt * tz1 * dz3)
    NPBMZ_LU_OFF(2, 3, (dt * tz2 * (u3 * tmp1)), )
    NPBMZ_LU_OFF(3, 0, (dt * tz2 * (-((u4 * tmp1) * (u4 * tmp1)) + 0.50e+00 * c2 * ((u2 * u2 + u3 * u3 + u4 * u4) *
                 tmp2))),
                 - dt * tz1 * (-r43 * c34 * tmp2 * u4))
    NPBMZ_LU_OFF(3, 1, (dt * tz2 * (-c2 * (u2 * tmp1))), )
    NPBMZ_LU_OFF(3, 2, (dt * tz2 * (-c2 * (u3 * tmp1))), )
    NPBMZ_LU_OFF(3, 3, (dt * tz2 * (2.0e+00 - c2) * (u4 * tmp1)), - dt * tz1 * (r43 * c34 * tmp1) - dt * tz1 * dz4)
    NPBMZ_LU_OFF(4, 0, (dt * tz2 * ((c2 * (u2 * u2 + u3 * u3 + u4 * u4) * tmp2 - c1 * (u5 * tmp1)) * (u4 * tmp1))),
                 - dt * tz1 * (-(c34 - c1345) * tmp3 * (u2 * u2) - (c34 - c1345) * tmp3 * (u3 * u3) - (r43 * c34 -
                 c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5))
    NPBMZ_LU_OFF(4, 1, (dt * tz2 * (-c2 * (u2 * u4) * tmp2)), - dt * tz1 * (c34 - c1345) * tmp2 * u2)
    NPBMZ_LU_OFF(4, 2, (dt * tz2 * (-c2 * (u3 * u4) * tmp2)), - dt * tz1 * (c34 - c1345) * tmp2 * u3)
    NPBMZ_LU_OFF(4, 3, (dt * tz2 * (c1 * (u5 * tmp1) - 0.50e+00 * c2 * ((u2 * u2 + u3 * u3 + 3.0e+00 * u4 * u4) *
                 tmp2))),
                 - dt * tz1 * (r43 * c34 - c1345) * tmp2 * u4)
    NPBMZ_LU_OFF(4, 4, (dt * tz2 * (c1 * (u4 * tmp1))), - dt * tz1 * c1345 * tmp1 - dt * tz1 * dz5)
  } else if (DIR == 1) {
    const double ty1 = J.ty1, ty2 = J.ty2;
    NPBMZ_LU_OFF(1, 0, (dt * ty2 * (-(u2 * u3) * tmp2)), - dt * ty1 * (-c34 * tmp2 * u2))
    NPBMZ_LU_OFF(1, 1, (dt * ty2 * (u3 * tmp1)), - dt * ty1 * (c34 * tmp1) - dt * ty1 * dy2)
    NPBMZ_LU_OFF(1, 2, (dt * ty2 * (u2 * tmp1)), )
    NPBMZ_LU_OFF(2, 0, (dt * ty2 * (-((u3 * tmp1) * (u3 * tmp1)) + 0.50e+00 * c2 * ((u2 * u2 + u3 * u3 + u4 * u4) *
                 tmp2))),
                 - dt * ty1 * (-r43 * c34 * tmp2 * u3))
    NPBMZ_LU_OFF(2, 1, (dt * ty2 * (-c2 * (u2 * tmp1))), )
    NPBMZ_LU_OFF(2, 2, (dt * ty2 * ((2.0e+00 - c2) * (u3 * tmp1))), - dt * ty1 * (r43 * c34 * tmp1) - dt * ty1 * dy3)
    NPBMZ_LU_OFF(2, 3, (dt * ty2 * (-c2 * (u4 * tmp1))), )
    NPBMZ_LU_OFF(3, 0, (dt * ty2 * (-(u3 * u4) * tmp2)), - dt * ty1 * (-c34 * tmp2 * u4))
    NPBMZ_LU_OFF(3, 2, (dt * ty2 * (u4 * tmp1)), )
    NPBMZ_LU_OFF(3, 3, (dt * ty2 * (u3 * tmp1)), - dt * ty1 * (c34 * tmp1) - dt * ty1 * dy4)
    NPBMZ_LU_OFF(4, 0, (dt * ty2 * ((c2 * (u2 * u2 + u3 * u3 + u4 * u4) * tmp2 - c1 * (u5 * tmp1)) * (u3 * tmp1))),
                 - dt * ty1 * (-(c34 - c1345) * tmp3 * (u2 * u2) - (r43 * c34 - c1345) * tmp3 * (u3 * u3) - (c34 -
                 c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5))
    NPBMZ_LU_OFF(4, 1, (dt * ty2 * (-c2 * (u2 * u3) * tmp2)), - dt * ty1 * (c34 - c1345) * tmp2 * u2)
    NPBMZ_LU_OFF(4, 2, (dt * ty2 * (c1 * (u5 * tmp1) - 0.50e+00 * c2 * ((u2 * u2 + 3.0e+00 * u3 * u3 + u4 * u4) *
                 tmp2))),
                 - dt * ty1 * (r43 * c34 - c1345) * tmp2 * u3)
    NPBMZ_LU_OFF(4, 3, (dt * ty2 * (-c2 * (u3 * u4) * tmp2)), - dt * ty1 * (c34 - c1345) * tmp2 * u4)
    NPBMZ_LU_OFF(4, 4, (dt * ty2 * (c1 * (u3 * tmp1))), - dt * ty1 * c1345 * tmp1 - dt * ty1 * dy5)
  } else {
    const double tx1 = J.tx1, tx2 = J.tx2;
    NPBMZ_LU_OFF(1, 0, (dt * tx2 * (-((u2 * tmp1) * (u2 * tmp1)) + c2 * 0.50e+00 * (u2 * u2 + u3 * u3 + u4 * u4) *
                 tmp2)),
                 - dt * tx1 * (-r43 * c34 * tmp2 * u2))
    NPBMZ_LU_OFF(1, 1, (dt * tx2 * ((2.0e+00 - c2) * (u2 * tmp1))), - dt * tx1 * (r43 * c34 * tmp1) - dt * tx1 * dx2)
    NPBMZ_LU_OFF(1, 2, (dt * tx2 * (-c2 * (u3 * tmp1))), )
    NPBMZ_LU_OFF(1, 3, (dt * tx2 * (-c2 * (u4 * tmp1))), )
    NPBMZ_LU_OFF(2, 0, (dt * tx2 * (-(u2 * u3) * tmp2)), - dt * tx1 * (-c34 * tmp2 * u3))
    NPBMZ_LU_OFF(2, 1, (dt * tx2 * (u3 * tmp1)), )
    NPBMZ_LU_OFF(2, 2, (dt * tx2 * (u2 * tmp1)), - dt * tx1 * (c34 * tmp1) - dt * tx1 * dx3)
    NPBMZ_LU_OFF(3, 0, (dt * tx2 * (-(u2 * u4) * tmp2)), - dt * tx1 * (-c34 * tmp2 * u4))
    NPBMZ_LU_OFF(3, 1, (dt * tx2 * (u4 * tmp1)), )
    NPBMZ_LU_OFF(3, 3, (dt * tx2 * (u2 * tmp1)), - dt * tx1 * (c34 * tmp1) - dt * tx1 * dx4)
    NPBMZ_LU_OFF(4, 0, (dt * tx2 * ((c2 * (u2 * u2 + u3 * u3 + u4 * u4) * tmp2 - c1 * (u5 * tmp1)) * (u2 * tmp1))),
                 - dt * tx1 * (-(r43 * c34 - c1345) * tmp3 * (u2 * u2) - (c34 - c1345) * tmp3 * (u3 * u3) - (c34 -
                 c1345) * tmp3 * (u4 * u4) - c1345 * tmp2 * u5))
    NPBMZ_LU_OFF(4, 1, (dt * tx2 * (c1 * (u5 * tmp1) - 0.50e+00 * c2 * ((3.0e+00 * u2 * u2 + u3 * u3 + u4 * u4) *
                 tmp2))),
                 - dt * tx1 * (r43 * c34 - c1345) * tmp2 * u2)
    NPBMZ_LU_OFF(4, 2, (dt * tx2 * (-c2 * (u3 * u2) * tmp2)), - dt * tx1 * (c34 - c1345) * tmp2 * u3)
    NPBMZ_LU_OFF(4, 3, (dt * tx2 * (-c2 * (u4 * u2) * tmp2)), - dt * tx1 * (c34 - c1345) * tmp2 * u4)
    NPBMZ_LU_OFF(4, 4, (dt * tx2 * (c1 * (u2 * tmp1))), - dt * tx1 * c1345 * tmp1 - dt * tx1 * dx5)
  }
#undef NPBMZ_LU_OFF
}

__device__ __forceinline__ void load5(const double* f, long long NP, long long p, double v[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m) v[m] = f[m * NP + p];
}

template <int DIR, int S>
__device__ __forceinline__ void store_blk(double* jac, long long NP, long long h, const double b[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (off_stored(DIR, r, c)) jac[(FAC_BLK + (2 * DIR + S) * BLK_N + blk_idx(DIR, r, c)) * NP + h] = b[r][c];
}

// Both blocks of direction DIR built from this point's state, stored at the
// interior consumers: the point at +1 in DIR reads jacld's, the point at -1
// jacu's.
template <int DIR>
__device__ __forceinline__ void jac_dir(const JC& J, double r1, const double u[5], double* __restrict__ jac,
                                        long long NP, bool lo, long long slot_lo, bool up, long long slot_up) {
  double b[5][5], c[5][5];
  jac_off<DIR>(J, r1, u[1], u[2], u[3], u[4], b, c);
  if (lo) store_blk<DIR, 0>(jac, NP, slot_lo, b);
  if (up) store_blk<DIR, 1>(jac, NP, slot_up, c);
}

// Slot of interior point (i, j, k) in the zone's hyperplane order (R: its row
// table, [l][k], ks entries per l).
__device__ __forceinline__ long long hp_slot(const LuZone& Z, const int* __restrict__ R, int ks, int i, int j, int k) {
  const int l = i + j + k;
  return Z.off + R[(long long)l * ks + k] + (j - max(2, l - k - (Z.nx - 1)));
}

// The inverse table of the sweeps: slot -> the point's index within its zone.
__global__ void __launch_bounds__(TPB) k_lu_points(LuDev D, const int* __restrict__ ri, int ls, int ks,
                                                   int* __restrict__ pts, const LuWork* __restrict__ work) {
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  int i, j, k;
  const int q = w.first + threadIdx.x;
  if (!decode(Z, q, i, j, k) || !interior(Z, i, j, k)) return;
  pts[hp_slot(Z, ri + (long long)w.zone * ls * ks, ks, i, j, k)] = q;
}

// jacld's and jacu's blocks and d's factors (the Jacobian work of ssor,
// taken off the wavefront): one thread per point of the zones (blockIdx.y:
// zone - z0), in the zone's full-box hyperplane order (i+j+k, then k, then
// j), so that consecutive threads write consecutive consumer slots.
// fb: per zone, l and k, the first full-box point of row k of hyperplane l;
// ri: the same for the interior points (the consumers' slots).
// Bound by the FP64 pipe.  480x320x28, us without / with contraction: 4913 /
// 4400 with jacld's and jacu's entries formed apart and a branch per missing
// consumer, 4343 / 3535 with each term formed once, 3705 / 3190 with the three
// directions of every point together (their squares and products shared).
// The zone's natural order instead of the hyperplane order (coalesced reads,
// scattered writes) costs 4670 / 4614 where this order takes 4343 / 3535.
__global__ void __launch_bounds__(TPB) k_lu_jac(LuDev D, const int* __restrict__ fb, int fls, const int* __restrict__ ri,
                                                int ls, int ks, double* __restrict__ jac, int z0) {
  const int zone = z0 + blockIdx.y;
  const LuZone Z = D.zones[zone];
  const int T = blockIdx.x * TPB + threadIdx.x;
  if (T >= Z.np) return;
  const int* FB = fb + (long long)zone * fls * ks;
  int lo = 3, hi = Z.nx + Z.ny + Z.nz;  // the hyperplane: largest l starting at or before T
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (FB[mid * ks] <= T) lo = mid; else hi = mid - 1;
  }
  const int l = lo;
  int klo = 1, khi = Z.nz;  // the row: largest k starting at or before T
  while (klo < khi) {
    const int mid = (klo + khi + 1) / 2;
    if (FB[l * ks + mid] <= T) klo = mid; else khi = mid - 1;
  }
  const int k = klo, j = max(1, l - k - Z.nx) + (T - FB[l * ks + k]), i = l - j - k;
  const long long NP = D.NP, p = pidx(Z, i, j, k);
  const JC J{D.dt, Z.tx1, Z.tx2, Z.ty1, Z.ty2, Z.tz1, Z.tz2};
  const int* R = ri + (long long)zone * ls * ks;
  auto slot = [&](int a, int b, int c) -> long long { return hp_slot(Z, R, ks, a, b, c); };
  const double r1 = D.prim[PR_RHO * NP + p];
  double u[5];
  load5(D.u, NP, p, u);
  const bool ii = i >= 2 && i <= Z.nx - 1, jj = j >= 2 && j <= Z.ny - 1, kk = k >= 2 && k <= Z.nz - 1;
  // every point forms the blocks of the three directions (the shared products
  // once), and stores those that have a consumer
  {
    const bool lo = jj && kk && i <= Z.nx - 2, up = jj && kk && i >= 3;
    jac_dir<0>(J, r1, u, jac, NP, lo, lo ? slot(i + 1, j, k) : 0, up, up ? slot(i - 1, j, k) : 0);
  }
  {
    const bool lo = ii && kk && j <= Z.ny - 2, up = ii && kk && j >= 3;
    jac_dir<1>(J, r1, u, jac, NP, lo, lo ? slot(i, j + 1, k) : 0, up, up ? slot(i, j - 1, k) : 0);
  }
  {
    const bool lo = ii && jj && k <= Z.nz - 2, up = ii && jj && k >= 3;
    jac_dir<2>(J, r1, u, jac, NP, lo, lo ? slot(i, j, k + 1) : 0, up, up ? slot(i, j, k - 1) : 0);
  }
  if (ii && jj && kk) {
    const long long h = slot(i, j, k);
    double b[5][5];
    jac_d(J, r1, u[1], u[2], u[3], u[4], b);
    const double rinv0 = 1.0e+00 / b[0][0];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      jac[(FAC_T + r) * NP + h] = b[r][r];
      jac[(FAC_Y + r) * NP + h] = 1.0e+00 / b[r][r];
    }
#pragma unroll
    for (int r = 1; r < 5; ++r) jac[(FAC_R0 + r - 1) * NP + h] = rinv0 * b[r][0];
#pragma unroll
    for (int c = 1; c <= 3; ++c) jac[(FAC_4C + c - 1) * NP + h] = (1.0e+00 / b[c][c]) * b[4][c];
  }
}

// ---- the wavefront sweeps (src/LU/blts.jl, src/LU/buts.jl) ------------------
// The entries of a zone's off-diagonal blocks that do not depend on the state,
// by the reference's expressions: [dir] k00 = -dt t1 d, kn = -+dt t2,
// k4 = -+dt t2 c2 (S = 0 jacld's signs, S = 1 jacu's).
struct RowConsts {
  double k00[3], kn[3], k4[3];
};
template <int S>
__device__ __forceinline__ RowConsts row_consts(double dt, const LuZone& Z) {
  RowConsts K;
  K.k00[0] = -dt * Z.tx1 * dx1;
  K.k00[1] = -dt * Z.ty1 * dy1;
  K.k00[2] = -dt * Z.tz1 * dz1;
  const double t2[3] = {Z.tx2, Z.ty2, Z.tz2};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    K.kn[d] = S == 0 ? -dt * t2[d] : dt * t2[d];
    K.k4[d] = S == 0 ? -dt * t2[d] * c2 : dt * t2[d] * c2;
  }
  return K;
}

// What row M of one point needs besides rsd: its rows of the three
// off-diagonal blocks and its part of d's factors.
struct RowCoef {
  double b[3][5];
  double f[4];  // rows 1..3: f[0] = tmp_m0; row 4: tmp_40, tmp_41, tmp_42, tmp_43
  double t, y;  // t_mm, 1 / t_mm
};

// Read-only load that stays where it is written: before the wait for the
// previous hyperplane (the compiler would sink a plain one to its use).
__device__ __forceinline__ double ld_early(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

template <int S, int M>
__device__ __forceinline__ void load_row(const double* __restrict__ jac, long long NP, long long h,
                                         const RowConsts& K, RowCoef& c) {
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int e = 0; e < 5; ++e) {
      if (off_zero(d, M, e)) continue;
      if (off_const(d, M, e))
        c.b[d][e] = M == 0 ? (e == 0 ? K.k00[d] : K.kn[d]) : K.k4[d];
      else
        c.b[d][e] = ld_early(jac + (FAC_BLK + (2 * d + S) * BLK_N + blk_idx(d, M, e)) * NP + h);
    }
  if (M > 0) c.f[0] = ld_early(jac + (FAC_R0 + M - 1) * NP + h);
  if (M == 4) {
#pragma unroll
    for (int q = 1; q <= 3; ++q) c.f[q] = ld_early(jac + (FAC_4C + q - 1) * NP + h);
  }
  c.t = ld_early(jac + (FAC_T + M) * NP + h);
  c.y = ld_early(jac + (FAC_Y + M) * NP + h);
}

// Row M of block z dotted with wz, summed left to right as the reference does
// (structural zeros skipped: a product with one is +-0 and adding it changes
// no sum's value).
template <int M>
__device__ __forceinline__ double row_dot_z(const RowCoef& c, const double wz[5]) {
  double s = 0.0;
  bool first = true;
#pragma unroll
  for (int e = 0; e < 5; ++e) {
    if (off_zero(2, M, e)) continue;
    const double t = c.b[2][e] * wz[e];
    s = first ? t : s + t;
    first = false;
  }
  return s;
}

// sum over e of Y[M][e] wy[e] + X[M][e] wx[e] (y term first, as blts / buts
// write it)
template <int M>
__device__ __forceinline__ double row_dot_yx(const RowCoef& c, const double wy[5], const double wx[5]) {
  double s = 0.0;
  bool first = true;
#pragma unroll
  for (int e = 0; e < 5; ++e) {
    if (!off_zero(1, M, e)) {
      const double t = c.b[1][e] * wy[e];
      s = first ? t : s + t;
      first = false;
    }
    if (!off_zero(0, M, e)) {
      const double t = c.b[0][e] * wx[e];
      s = first ? t : s + t;
      first = false;
    }
  }
  return s;
}

// Row M of one point of a sweep (UP false: blts, the neighbours at -1; UP
// true: buts, the neighbours at +1); h: the point's slot, -1 for a lane
// without one.  SCALE: rsd *= dt at the point first (ssor's scaling, fused:
// blts reads only points it has already scaled and solved, or boundary
// points, which it does not touch).
template <bool UP, bool SCALE, int M>
__device__ __forceinline__ void sweep_row(const LuDev& D, const LuSweep& S, const LuZone& Z, long long h, int lane,
                                          double (*sv)[HP]) {
  const long long NP = D.NP;
  RowCoef c;
  long long p = 0;
  if (h >= 0) {
    p = Z.off + __ldg(S.pts + h);
    load_row<UP ? 1 : 0, M>(S.jac, NP, h, row_consts<UP ? 1 : 0>(D.dt, Z), c);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous hyperplane's rsd from here on
  double own = 0.0, v = 0.0;
  if (h >= 0) {
    const long long sgn = UP ? 1 : -1, sy = sgn * Z.nx, sz = sy * Z.ny;
    double wz[5], wy[5], wx[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double* r = D.rsd + m * NP + p;
      wz[m] = __ldcg(r + sz);
      wy[m] = __ldcg(r + sy);
      wx[m] = __ldcg(r + sgn);
    }
    own = __ldcg(D.rsd + M * NP + p);
    const double omega = D.omega;
    if (!UP) {
      v = SCALE ? D.dt * own : own;
      v = v - omega * row_dot_z<M>(c, wz);
      v = v - omega * row_dot_yx<M>(c, wy, wx);
    } else {
      v = omega * row_dot_z<M>(c, wz);
      v = v + omega * row_dot_yx<M>(c, wy, wx);
    }
  }
  // the solve with d: rows 1..4 subtract v_0's part, then row 4 that of 1..3
  if (M == 0) sv[0][lane] = v;
  __syncthreads();
  if (M > 0 && h >= 0) v = v - sv[0][lane] * c.f[0];
  if (M > 0 && M < 4) sv[M][lane] = v;
  __syncthreads();
  if (h < 0) return;
  if (M == 4) {
#pragma unroll
    for (int r = 1; r <= 3; ++r) v = v - sv[r][lane] * c.f[r];
  }
  v = div_y(v, c.t, c.y);
  D.rsd[M * NP + p] = UP ? own - v : v;
}

// blts (UP false) / buts (UP true) at the points of hyperplane i+j+k = l of
// zones z0 + blockIdx.y, five threads per point: one warp per row and HP
// points.  Launched once per hyperplane, each launch a programmatic dependent
// of the one before: its blocks take their place and fetch the coefficients,
// which the sweep does not change, while the previous hyperplane still runs,
// and wait for it before they read rsd.
// Bound: an SM quarter takes an FP64 warp instruction every 64 cycles whatever
// its active lanes, so the longest row's chain (45 FP64 instructions for row 4
// without contraction) sets the time of a small hyperplane, and the sum of
// the rows (171 a point) that of a large one.  Rows 0 and 1, the
// cheapest, run on warps 0 and 4, which share an SM quarter.
// Both sweeps of one iteration (us, with block rows of 32 points, separate
// loads and no overlap of the launches, and now): 64x64x8
// 576 / 193, 304x208x17 contracted 3184 / 1456, 480x320x28 8180 / 4130.  One
// launch for a whole sweep with one thread-block cluster per zone and cluster
// barriers between the hyperplanes took 222, 1820 and 7150 there: a zone has
// eight SMs then.
template <bool UP, bool SCALE>
__global__ void __launch_bounds__(HP * 5, 4) k_lu_sweep(LuDev D, LuSweep S, int l, int z0) {
  __shared__ double sv[4][HP];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int zone = z0 + blockIdx.y, lane = threadIdx.x, t = blockIdx.x * HP + lane;
  const LuZone Z = D.zones[zone];
  const int* hps = S.hps + (long long)zone * S.hstride + l;
  const int lo = __ldg(hps), n = __ldg(hps + 1) - lo;
  const long long h = t < n ? Z.off + lo + t : -1;
  switch (threadIdx.y) {
    case 0: sweep_row<UP, SCALE, 0>(D, S, Z, h, lane, sv); break;
    case 1: sweep_row<UP, SCALE, 4>(D, S, Z, h, lane, sv); break;
    case 2: sweep_row<UP, SCALE, 2>(D, S, Z, h, lane, sv); break;
    case 3: sweep_row<UP, SCALE, 3>(D, S, Z, h, lane, sv); break;
    default: sweep_row<UP, SCALE, 1>(D, S, Z, h, lane, sv); break;
  }
}

__device__ inline void face_sizes(const LuZone& Z, int nkp, long long& e, long long& s) {
  e = (long long)Z.nx * nkp;
  s = (long long)Z.ny * nkp;
}

__global__ void __launch_bounds__(TPB) k_lu_pack(LuDev D, Faces F, int nzones) {
  const int z = blockIdx.y;
  if (z >= nzones) return;
  const LuZone Z = D.zones[z];
  const int per = 2 * Z.nx + 2 * Z.ny;
  const int t = blockIdx.x * TPB + threadIdx.x;
  if (t >= per * F.nkp) return;
  const int kq = t / per, pos = t % per, k = F.klo + kq;
  long long ne, ns;
  face_sizes(Z, F.nkp, ne, ns);
  double* base = F.stage + F.zoff[z];
  int i, j;
  long long so;
  if (pos < Z.nx) {  // east face
    i = pos + 1; j = Z.ny - 1; so = 0 * ne + (long long)kq * Z.nx + pos;
  } else if (pos < 2 * Z.nx) {  // west face
    i = pos - Z.nx + 1; j = 2; so = 5 * ne + (long long)kq * Z.nx + (pos - Z.nx);
  } else if (pos < 2 * Z.nx + Z.ny) {  // south face
    i = Z.nx - 1; j = pos - 2 * Z.nx + 1; so = 10 * ne + (long long)kq * Z.ny + (j - 1);
  } else {  // north face
    i = 2; j = pos - 2 * Z.nx - Z.ny + 1; so = 10 * ne + 5 * ns + (long long)kq * Z.ny + (j - 1);
  }
  const long long p = pidx(Z, i, j, k);
  const long long stride = pos < 2 * Z.nx ? ne : ns;
#pragma unroll
  for (int m = 0; m < 5; ++m) base[so + m * stride] = D.u[m * D.NP + p];
}

// Every ghost point has one writer: j = 1 / j = ny (west / east) include the
// corners, which the reference's unpack order (south, north, west, east)
// leaves to them.
__global__ void __launch_bounds__(TPB) k_lu_unpack(LuDev D, Faces F, int nzones) {
  const int z = blockIdx.y;
  if (z >= nzones) return;
  const LuZone Z = D.zones[z];
  const int per = 2 * Z.nx + 2 * (Z.ny - 2);
  const int t = blockIdx.x * TPB + threadIdx.x;
  if (t >= per * F.nkp) return;
  const int kq = t / per, pos = t % per, k = F.klo + kq;
  int i, j, src;
  long long so, stride;
  if (pos < Z.nx) {  // west ghost j = 1 <- west zone's east face
    i = pos + 1; j = 1; src = F.nbr[4 * z + 0];
    const LuZone S = D.zones[src];
    long long ne, ns;
    face_sizes(S, F.nkp, ne, ns);
    so = F.zoff[src] + 0 * ne + (long long)kq * S.nx + (i - 1); stride = ne;
  } else if (pos < 2 * Z.nx) {  // east ghost j = ny <- east zone's west face
    i = pos - Z.nx + 1; j = Z.ny; src = F.nbr[4 * z + 1];
    const LuZone S = D.zones[src];
    long long ne, ns;
    face_sizes(S, F.nkp, ne, ns);
    so = F.zoff[src] + 5 * ne + (long long)kq * S.nx + (i - 1); stride = ne;
  } else if (pos < 2 * Z.nx + (Z.ny - 2)) {  // north ghost i = 1 <- north zone's south face
    i = 1; j = pos - 2 * Z.nx + 2; src = F.nbr[4 * z + 3];
    const LuZone S = D.zones[src];
    long long ne, ns;
    face_sizes(S, F.nkp, ne, ns);
    so = F.zoff[src] + 10 * ne + (long long)kq * S.ny + (j - 1); stride = ns;
  } else {  // south ghost i = nx <- south zone's north face
    i = Z.nx; j = pos - 2 * Z.nx - (Z.ny - 2) + 2; src = F.nbr[4 * z + 2];
    const LuZone S = D.zones[src];
    long long ne, ns;
    face_sizes(S, F.nkp, ne, ns);
    so = F.zoff[src] + 10 * ne + 5 * ns + (long long)kq * S.ny + (j - 1); stride = ns;
  }
  const long long p = pidx(Z, i, j, k);
  double g[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    g[m] = F.stage[so + m * stride];
    D.u[m * D.NP + p] = g[m];
  }
  store_prim(D.prim, D.NP, p, g);
}

// ---- norms (src/LU/l2norm.jl, src/LU/error.jl, src/LU/pintgr.jl) -----------
// WHICH 0: sum of rsd^2, 1: sum of (exact - u)^2 over the interior; one row
// of 5 partial sums per work block (fixed-order tree reduction)
template <int WHICH>
__global__ void __launch_bounds__(TPB) k_lu_norm_partial(LuDev D, const LuWork* __restrict__ work, CeTable ce,
                                                         double* partial) {
  __shared__ double sh[5][TPB];
  const LuWork w = work[blockIdx.x];
  const LuZone Z = D.zones[w.zone];
  double s[5] = {0, 0, 0, 0, 0};
  int i, j, k;
  if (decode(Z, w.first + threadIdx.x, i, j, k) && interior(Z, i, j, k)) {
    const long long p = pidx(Z, i, j, k);
    if (WHICH == 0) {
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        const double r = D.rsd[m * D.NP + p];
        s[m] = r * r;
      }
    } else {
      double e[5];
      exact_point(ce, i, j, k, Z.nx, Z.ny, Z.nz, e);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        const double t = e[m] - D.u[m * D.NP + p];
        s[m] = t * t;
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) sh[m][threadIdx.x] = s[m];
  __syncthreads();
  for (int h = TPB / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h)
#pragma unroll
      for (int m = 0; m < 5; ++m) sh[m][threadIdx.x] += sh[m][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x < 5) partial[(long long)blockIdx.x * 5 + threadIdx.x] = sh[threadIdx.x][0];
}

// per zone: sqrt(sum / ((nx-2)(ny-2)(nz-2))), then summed over zones in
// order into out[5] (+ out_zone[5*z + m] when non-null); one thread per m
__global__ void k_lu_norm_finish(const LuZone* zones, const int* zblock, int nzones, const double* partial,
                                 double* out, double* out_zone) {
  const int m = threadIdx.x;
  if (m >= 5) return;
  double total = 0.0;
  for (int z = 0; z < nzones; ++z) {
    double s = 0.0;
    for (int b = zblock[z]; b < zblock[z + 1]; ++b) s += partial[(long long)b * 5 + m];
    const LuZone Z = zones[z];
    const double r = sqrt(s / ((double)(Z.nx - 2) * (Z.ny - 2) * (Z.nz - 2)));
    if (out_zone) out_zone[5 * z + m] = r;
    total += r;
  }
  out[m] = total;
}

// pintgr of one zone per block (one process: ibeg = ii1, ifin = ii2,
// jbeg = ji1, jfin = ji2); frc[z] = 0.25 (frc1 + frc2 + frc3)
__global__ void __launch_bounds__(TPB) k_lu_pintgr(LuDev D, double* frc) {
  __shared__ double sh[3][TPB];
  const LuZone Z = D.zones[blockIdx.x];
  const int ibeg = ii1, ifin = Z.ii2, jbeg = ji1, jfin = Z.ji2, ifin1 = ifin - 1, jfin1 = jfin - 1;
  auto phi = [&](int i, int j, int k) {
    const long long p = pidx(Z, i, j, k);
    const double u1 = D.u[p], u2 = D.u[D.NP + p], u3 = D.u[2 * D.NP + p], u4 = D.u[3 * D.NP + p],
                 u5 = D.u[4 * D.NP + p];
    return c2 * (u5 - 0.50e+00 * (u2 * u2 + u3 * u3 + u4 * u4) / u1);
  };
  double s1 = 0.0, s2 = 0.0, s3 = 0.0;
  const int n1i = ifin1 - ibeg + 1, n1j = jfin1 - jbeg + 1, nk = Z.ki2 - 1 - ki1 + 1;
  for (int t = threadIdx.x; t < n1i * n1j; t += TPB) {
    const int i = ibeg + t % n1i, j = jbeg + t / n1i;
    s1 += (phi(i, j, ki1) + phi(i + 1, j, ki1) + phi(i, j + 1, ki1) + phi(i + 1, j + 1, ki1) + phi(i, j, Z.ki2) +
           phi(i + 1, j, Z.ki2) + phi(i, j + 1, Z.ki2) + phi(i + 1, j + 1, Z.ki2));
  }
  for (int t = threadIdx.x; t < n1i * nk; t += TPB) {
    const int i = ibeg + t % n1i, k = ki1 + t / n1i;
    s2 += (phi(i, jbeg, k) + phi(i + 1, jbeg, k) + phi(i, jbeg, k + 1) + phi(i + 1, jbeg, k + 1) + phi(i, jfin, k) +
           phi(i + 1, jfin, k) + phi(i, jfin, k + 1) + phi(i + 1, jfin, k + 1));
  }
  for (int t = threadIdx.x; t < n1j * nk; t += TPB) {
    const int j = jbeg + t % n1j, k = ki1 + t / n1j;
    s3 += (phi(ibeg, j, k) + phi(ibeg, j + 1, k) + phi(ibeg, j, k + 1) + phi(ibeg, j + 1, k + 1) + phi(ifin, j, k) +
           phi(ifin, j + 1, k) + phi(ifin, j, k + 1) + phi(ifin, j + 1, k + 1));
  }
  sh[0][threadIdx.x] = s1;
  sh[1][threadIdx.x] = s2;
  sh[2][threadIdx.x] = s3;
  __syncthreads();
  for (int h = TPB / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h)
      for (int q = 0; q < 3; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double frc1 = Z.dxi * Z.deta * sh[0][0];
    const double frc2 = Z.dxi * Z.dzeta * sh[1][0];
    const double frc3 = Z.deta * Z.dzeta * sh[2][0];
    frc[blockIdx.x] = 0.25e+00 * (frc1 + frc2 + frc3);
  }
}

// ---- layout conversion --------------------------------------------------------
// REF: [1:5, -1:nx+2, -1:ny+2, 1:nz] column-major; DENSE: [m][k][j][i].  One
// thread per double, in the host array's order (REF: the 5*nx interior
// doubles of each (j, k) row are contiguous), so that a warp's host accesses
// are contiguous: the host side may be page-locked memory read or written
// in place over the host link.
template <bool REF, bool TO_DEV>
__global__ void __launch_bounds__(TPB) k_lu_convert(LuDev D, double* field, double* host_img, int zone) {
  const LuZone Z = D.zones[zone];
  const long long t = (long long)blockIdx.x * TPB + threadIdx.x;
  if (t >= 5LL * Z.np) return;
  int m, i, j, k;
  long long h;
  if (REF) {
    const int rowlen = 5 * Z.nx;
    const int row = (int)(t / rowlen), e = (int)(t % rowlen);
    m = e % 5;
    i = e / 5 + 1;
    j = row % Z.ny + 1;
    k = row / Z.ny + 1;
    h = 5LL * (Z.nx + 4) * ((j + 1) + (long long)(Z.ny + 4) * (k - 1)) + 10 + e;
  } else {
    m = (int)(t / Z.np);
    const int q = (int)(t % Z.np);
    i = q % Z.nx + 1;
    j = (q / Z.nx) % Z.ny + 1;
    k = q / (Z.nx * Z.ny) + 1;
    h = t;
  }
  const long long p = m * D.NP + pidx(Z, i, j, k);
  if (TO_DEV)
    field[p] = host_img[h];
  else
    host_img[h] = field[p];
}

// ---- host launchers ------------------------------------------------------------
void rhs(bool erhs, const LuDev& D, const LuWork* w, int n, const double* g, const double* prim, double* out,
         cudaStream_t s) {
  if (erhs)
    k_lu_rhs<true><<<n, TPB, 0, s>>>(D, w, g, prim, out);
  else
    k_lu_rhs<false><<<n, TPB, 0, s>>>(D, w, g, prim, out);
}
void init(const LuDev& D, const LuWork* w, int n, const CeTable& ce, cudaStream_t s) {
  k_lu_init<<<n, TPB, 0, s>>>(D, w, ce);
}
void poly(const LuDev& D, const LuWork* w, int n, const CeTable& ce, cudaStream_t s) {
  k_lu_poly<<<n, TPB, 0, s>>>(D, w, ce);
}
void prim(const LuDev& D, const LuWork* w, int n, const double* g, cudaStream_t s) {
  k_lu_prim<<<n, TPB, 0, s>>>(D, w, g);
}
void pointwise(bool update, const LuDev& D, const LuWork* w, int n, double tmp, cudaStream_t s) {
  if (update)
    k_lu_pointwise<true><<<n, TPB, 0, s>>>(D, w, tmp);
  else
    k_lu_pointwise<false><<<n, TPB, 0, s>>>(D, w, tmp);
}
void jac(const LuDev& D, const int* fb, int fls, const int* ri, int ls, int ks, double* jac, int z0, dim3 grid,
         cudaStream_t s) {
  k_lu_jac<<<grid, TPB, 0, s>>>(D, fb, fls, ri, ls, ks, jac, z0);
}
void points(const LuDev& D, const int* ri, int ls, int ks, int* pts, const LuWork* w, int n, cudaStream_t s) {
  k_lu_points<<<n, TPB, 0, s>>>(D, ri, ls, ks, pts, w);
}
// follows: the launch before it in the stream is the hyperplane before it
cudaError_t sweep(bool up, bool scale, const LuDev& D, const LuSweep& S, int l, int z0, dim3 grid, bool follows,
                  cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  cfg.gridDim = grid;
  cfg.blockDim = dim3(HP, 5);
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = follows ? 1 : 0;
  if (up) return cudaLaunchKernelEx(&cfg, k_lu_sweep<true, false>, D, S, l, z0);
  if (scale) return cudaLaunchKernelEx(&cfg, k_lu_sweep<false, true>, D, S, l, z0);
  return cudaLaunchKernelEx(&cfg, k_lu_sweep<false, false>, D, S, l, z0);
}
void pack(const LuDev& D, const Faces& F, int nzones, dim3 grid, cudaStream_t s) {
  k_lu_pack<<<grid, TPB, 0, s>>>(D, F, nzones);
}
void unpack(const LuDev& D, const Faces& F, int nzones, dim3 grid, cudaStream_t s) {
  k_lu_unpack<<<grid, TPB, 0, s>>>(D, F, nzones);
}
void norm_partial(int which, const LuDev& D, const LuWork* w, int n, const CeTable& ce, double* partial,
                  cudaStream_t s) {
  if (which == 0)
    k_lu_norm_partial<0><<<n, TPB, 0, s>>>(D, w, ce, partial);
  else
    k_lu_norm_partial<1><<<n, TPB, 0, s>>>(D, w, ce, partial);
}
void norm_finish(const LuZone* zones, const int* zblock, int nzones, const double* partial, double* out,
                 cudaStream_t s) {
  k_lu_norm_finish<<<1, 32, 0, s>>>(zones, zblock, nzones, partial, out, nullptr);
}
void pintgr(const LuDev& D, int nzones, double* frc, cudaStream_t s) { k_lu_pintgr<<<nzones, TPB, 0, s>>>(D, frc); }
void convert(bool ref, bool to_dev, const LuDev& D, double* field, double* img, int zone, int blocks, cudaStream_t s) {
  if (ref && to_dev)
    k_lu_convert<true, true><<<blocks, TPB, 0, s>>>(D, field, img, zone);
  else if (ref)
    k_lu_convert<true, false><<<blocks, TPB, 0, s>>>(D, field, img, zone);
  else if (to_dev)
    k_lu_convert<false, true><<<blocks, TPB, 0, s>>>(D, field, img, zone);
  else
    k_lu_convert<false, false><<<blocks, TPB, 0, s>>>(D, field, img, zone);
}

}  // namespace LU_NS
}  // namespace npbmz_lu
