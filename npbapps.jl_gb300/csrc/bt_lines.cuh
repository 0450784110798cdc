// bt_lines.cuh -- the BT block-tridiagonal elimination of the FMA build
// (included by step_kernels.cuh inside its namespace; FP64 and FP32).
//
// The rows are the reference's (src/BT/x_solve.jl:536-708, y_solve.jl,
// z_solve.jl), with the scaled Jacobians G = tmp2 fjac and
// H = tmp1 (njac + diag(d)) of a point's state formed once:
//   -lhsa of the next point  P = G + H
//    lhsb of the point       B = I + 2 H
//    lhsc of the point before C = G - H
// so that a row is  x_p + ... : B' = B_p + P_{p-1} C'_{p-1},
// r' = r_p + P_{p-1} r'_{p-1}, and B' [C' r''] = [C_p r'].  B' is factored
// as L U with scaled pivot rows (U has a unit diagonal) instead of the
// reference's Gauss-Jordan form: 40 instead of 50 operations on B', the same
// on the right-hand sides.  The elimination visits the row of rho first, then
// the two tangential momenta, the normal momentum and the energy: the rows
// visited first have few nonzeros in C, whose zero columns are skipped until
// they fill.  One point takes 389 FP64 instructions (531 with the blocks
// formed entry by entry and Gauss-Jordan): five steps of 128x128x16 went from
// 11.16 to 9.17 ms.  The FP32 sweeps of 480x320x28 (whose second pass also no
// longer stores C' again) went from 640, 610 and 681 to 586, 568 and 635 us.
#pragma once

template <int DIR>
__host__ __device__ constexpr int bt_piv(int s) {  // the row eliminated at step s
  return s == 0 ? 0 : s == 4 ? 4 : s == 3 ? DIR + 1 : DIR == 0 ? s + 1 : DIR == 1 ? 2 * s - 1 : s;
}
template <int DIR>
__host__ __device__ constexpr int bt_rank(int c) {  // the step that eliminates row c
  for (int s = 0; s < 5; ++s)
    if (bt_piv<DIR>(s) == c) return s;
  return 5;
}
// Columns of C that are nonzero in the row of step s when it becomes the pivot
// row (its own nonzeros and what the earlier steps filled in); increasing in s.
template <int DIR>
__host__ __device__ constexpr bool bt_cset(int s, int c) {
  return s >= 3 || c == 0 || c == DIR + 1 || (s >= 1 && c == bt_piv<DIR>(1)) || (s >= 2 && c == bt_piv<DIR>(2));
}

// G and H of one point (structural nonzeros only) from 1/rho, the velocities,
// E = u5/rho and q = |v|^2 / 2.
template <int DIR, typename T>
__device__ __forceinline__ void bt_gh(const BtK<T>& k, T ri, const T v[3], T E, T q, T G[5][5], T H[5][5]) {
  constexpr int a = DIR + 1;
  const T vn = v[DIR];
  const T V[3] = {k.t2 * v[0], k.t2 * v[1], k.t2 * v[2]};
  const T Vn = V[DIR], X = k.c2t2 * q, Y = Vn * vn, e1 = k.c1t2 * E;
  G[0][a] = k.t2;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    if (m == DIR) continue;
    G[m + 1][0] = -(Vn * v[m]);
    G[m + 1][m + 1] = Vn;
    G[m + 1][a] = V[m];
    G[a][m + 1] = -(k.c2 * V[m]);
    G[4][m + 1] = G[a][m + 1] * vn;
  }
  G[a][0] = X - Y;
  G[a][a] = k.two_m_c2 * Vn;
  G[a][4] = k.c2t2;
  G[4][0] = fma((T)2.0, X, -e1) * vn;
  G[4][a] = fma(-k.c2, Y, e1 - X);
  G[4][4] = k.c1 * Vn;
  const T kt = k.kc * ri, kn = k.k43 * ri, g = k.kg * ri;
  const T wt = kt - g, wn = kn - g;
  H[0][0] = k.t1d[0];
  T s = g * E;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const T km = m == DIR ? kn : kt;
    H[m + 1][0] = -(km * v[m]);
    H[m + 1][m + 1] = km + k.t1d[m + 1];
    H[4][m + 1] = (m == DIR ? wn : wt) * v[m];
    s = fma(H[4][m + 1], v[m], s);
  }
  H[4][0] = -s;
  H[4][4] = g + k.t1d[4];
}

template <int DIR>
__host__ __device__ constexpr bool hnz(int r, int c) { return nnz(r, c) || (r == 0 && c == 0); }

template <int DIR, typename T>
__device__ __forceinline__ void bt_form_p(const T G[5][5], const T H[5][5], T P[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (anz<DIR>(r, c)) P[r][c] = !hnz<DIR>(r, c) ? G[r][c] : !fnz<DIR>(r, c) ? H[r][c] : G[r][c] + H[r][c];
}
template <int DIR, typename T>
__device__ __forceinline__ void bt_form_c(const T G[5][5], const T H[5][5], T C[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (anz<DIR>(r, c)) C[r][c] = !hnz<DIR>(r, c) ? G[r][c] : !fnz<DIR>(r, c) ? -H[r][c] : G[r][c] - H[r][c];
}
template <int DIR, typename T>
__device__ __forceinline__ void bt_form_b(const T H[5][5], T B[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (hnz<DIR>(r, c)) B[r][c] = r == c ? fma((T)2.0, H[r][c], (T)1.0) : (T)2.0 * H[r][c];
}

// Pivot reciprocal: FP64 by Newton-Raphson from the FP32 estimate (2 ulps),
// FP32 the fast reciprocal (the refinement corrects the solve).
__device__ __forceinline__ double bt_recip(double b) { return nr_rcp(b); }
__device__ __forceinline__ float bt_recip(float b) { return __fdividef(1.0f, b); }

// L U of B (unit-diagonal U, pivot reciprocals on the diagonal) applied to C
// (structural nonzeros on entry, full on exit) and r.
template <int DIR, typename T>
__device__ __forceinline__ void bt_factor_solve(T B[5][5], T C[5][5], T r[5]) {
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    constexpr int D = DIR;
    const int p = bt_piv<D>(s);
    const T piv = bt_recip(B[p][p]);
    B[p][p] = piv;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      if (bt_rank<D>(c) > s) B[p][c] *= piv;
      if (bt_cset<D>(s, c)) C[p][c] *= piv;
    }
    r[p] *= piv;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (bt_rank<D>(q) <= s) continue;
      const T m = B[q][p];
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        if (bt_rank<D>(c) > s) B[q][c] = fma(-m, B[p][c], B[q][c]);
        if (bt_cset<D>(s, c))
          C[q][c] = anz<D>(q, c) || (s > 0 && bt_cset<D>(s - 1, c)) ? fma(-m, C[p][c], C[q][c]) : -(m * C[p][c]);
      }
      r[q] = fma(-m, r[p], r[q]);
    }
  }
#pragma unroll
  for (int s = 4; s > 0; --s) {
    const int p = bt_piv<DIR>(s);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (bt_rank<DIR>(q) >= s) continue;
      const T m = B[q][p];
#pragma unroll
      for (int c = 0; c < 5; ++c)
        C[q][c] = s < 4 || bt_cset<DIR>(bt_rank<DIR>(q), c) ? fma(-m, C[p][c], C[q][c]) : -(m * C[p][c]);
      r[q] = fma(-m, r[p], r[q]);
    }
  }
}

// The same factors applied to r alone.
template <int DIR, typename T>
__device__ __forceinline__ void bt_apply_factors(const T B[5][5], T r[5]) {
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int p = bt_piv<DIR>(s);
    r[p] *= B[p][p];
#pragma unroll
    for (int q = 0; q < 5; ++q)
      if (bt_rank<DIR>(q) > s) r[q] = fma(-B[q][p], r[p], r[q]);
  }
#pragma unroll
  for (int s = 4; s > 0; --s) {
    const int p = bt_piv<DIR>(s);
#pragma unroll
    for (int q = 0; q < 5; ++q)
      if (bt_rank<DIR>(q) < s) r[q] = fma(-B[q][p], r[p], r[q]);
  }
}

// r += P x
template <int DIR, typename T>
__device__ __forceinline__ void bt_add_px(const T P[5][5], const T x[5], T r[5]) {
#pragma unroll
  for (int m = 0; m < 5; ++m)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (anz<DIR>(m, c)) r[m] = fma(P[m][c], x[c], r[m]);
}

// B' = B + P C' (B structural on entry, full on exit)
template <int DIR, typename T>
__device__ __forceinline__ void bt_add_pc(const T P[5][5], const T Cp[5][5], const T Bs[5][5], T B[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      T t = hnz<DIR>(r, c) ? Bs[r][c] : (T)0.0;
#pragma unroll
      for (int e = 0; e < 5; ++e)
        if (anz<DIR>(r, e)) t = fma(P[r][e], Cp[e][c], t);
      B[r][c] = t;
    }
}

// State of one point for bt_gh from the primitive planes.
template <typename T>
struct BtState {
  T ri, v[3], u5, q;
};
template <typename T>
__device__ __forceinline__ BtState<T> bt_load_state(const Fields& F, int64_t pt) {
  const int64_t NP = F.NP;
  BtState<T> s;
  s.ri = (T)F.prim[PR_RHOI * NP + pt];
  s.v[0] = (T)F.prim[PR_US * NP + pt];
  s.v[1] = (T)F.prim[PR_VS * NP + pt];
  s.v[2] = (T)F.prim[PR_WS * NP + pt];
  s.q = (T)F.prim[PR_QS * NP + pt];
  s.u5 = (T)F.u[4 * NP + pt];
  return s;
}

// The line solve, one thread per line (src/BT/x_solve.jl:444-488,501-1746 and
// its y, z copies): C'_p goes to the line scratch lhsc[(p*25 + e) * nlt +
// line], the eliminated rhs back into rhs.  The next point's state and rhs
// are loaded one step ahead.
template <int DIR, typename T>
__global__ void __launch_bounds__(128) k_bt_line(Fields F, Consts K, const Work* __restrict__ work,
                                                 T* __restrict__ lhsc, int64_t nlt, int add_u) {
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
  const BtK<T>& k = bt_consts<T>(K, DIR);
  T rp[5], Cp[5][5], Pcur[5][5], Pnext[5][5], Bs[5][5], G[5][5], H[5][5];
  BtState<T> s = bt_load_state<T>(F, base);
  bt_gh<DIR, T>(k, s.ri, s.v, s.u5 * s.ri, s.q, G, H);
  bt_form_p<DIR, T>(G, H, Pcur);
  s = bt_load_state<T>(F, base + st);
  bt_gh<DIR, T>(k, s.ri, s.v, s.u5 * s.ri, s.q, G, H);
  bt_form_p<DIR, T>(G, H, Pnext);
  bt_form_b<DIR, T>(H, Bs);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    rp[m] = (T)rhs[m * NP + base];
#pragma unroll
    for (int c = 0; c < 5; ++c) Cp[m][c] = (T)0.0;
  }
  T rn[5];
  s = bt_load_state<T>(F, base + 2 * st);
#pragma unroll
  for (int m = 0; m < 5; ++m) rn[m] = (T)rhs[m * NP + base + st];
  for (int p = 1; p <= n - 2; ++p) {
    const int64_t pt = base + p * st;
    T r[5], B[5][5], C[5][5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = rn[m];
    const BtState<T> sp = s;
    if (p + 2 <= n - 1) {
      s = bt_load_state<T>(F, pt + 2 * st);
#pragma unroll
      for (int m = 0; m < 5; ++m) rn[m] = (T)rhs[m * NP + pt + st];
    }
    bt_add_px<DIR, T>(Pcur, rp, r);
    bt_add_pc<DIR, T>(Pcur, Cp, Bs, B);
    bt_gh<DIR, T>(k, sp.ri, sp.v, sp.u5 * sp.ri, sp.q, G, H);
    bt_form_c<DIR, T>(G, H, C);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b)
        if (anz<DIR>(a, b)) Pcur[a][b] = Pnext[a][b];
    bt_form_p<DIR, T>(G, H, Pnext);
    bt_form_b<DIR, T>(H, Bs);
    bt_factor_solve<DIR, T>(B, C, r);
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
      rhs[m * NP + pt] = (double)r[m];
    }
  }
  // back substitution: x_p = r'_p - C'_p x_{p+1}; the last point is its rhs
#pragma unroll
  for (int m = 0; m < 5; ++m) rn[m] = (T)rhs[m * NP + base + (n - 1) * st];
  for (int p = n - 2; p >= 1; --p) {
    const int64_t pt = base + p * st;
    T r[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) r[m] = (p == n - 2) ? rp[m] : (T)rhs[m * NP + pt];
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
      for (int c = 0; c < 5; ++c) r[m] = fma(-lhsc[((int64_t)p * 25 + m * 5 + c) * nlt + gl], rn[c], r[m]);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double v = (double)r[m];
      rhs[m * NP + pt] = v;
      if (add_u) F.u[m * NP + pt] += v;
      rn[m] = r[m];
    }
  }
}
