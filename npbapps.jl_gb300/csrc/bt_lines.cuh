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
// they fill.  One point takes 302 to 308 FP64 instructions (about 480 with the
// blocks formed entry by entry and Gauss-Jordan): five steps of 128x128x16 went
// from 11.16 to 9.17 ms.  The FP32 sweeps of 480x320x28 (whose second pass also no
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

// Products and sums that the compiler does not contract.
__device__ __forceinline__ double bt_mul(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ float bt_mul(float x, float y) { return __fmul_rn(x, y); }
__device__ __forceinline__ double bt_add(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ float bt_add(float x, float y) { return __fadd_rn(x, y); }

// Entries of G that are one product, multiplied when P and C are formed.
template <int DIR>
__host__ __device__ constexpr bool gprod(int r, int c) {
  return r == 4 ? c != DIR + 1 : r == DIR + 1 ? c == r : r > 0 && c == 0;
}
template <int DIR>
__host__ __device__ constexpr bool hnz(int r, int c) { return nnz(r, c) || (r == 0 && c == 0); }

// G (gprod entries: G * Gb) and H of one point (structural nonzeros only) from
// 1/rho, the velocities, E = u5/rho and q = |v|^2 / 2.
template <int DIR, typename T>
struct BtGH {
  T G[5][5], Gb[5][5], H[5][5];
};
template <int DIR, typename T>
__device__ __forceinline__ void bt_gh(const BtK<T>& k, T ri, const T v[3], T E, T q, BtGH<DIR, T>& o) {
  constexpr int a = DIR + 1;
  const T vn = v[DIR];
  const T V[3] = {bt_mul(k.t2, v[0]), bt_mul(k.t2, v[1]), bt_mul(k.t2, v[2])};
  const T Vn = V[DIR], X = bt_mul(k.c2t2, q), Y = bt_mul(Vn, vn), e1 = bt_mul(k.c1t2, E);
  o.G[0][a] = k.t2;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    if (m == DIR) continue;
    o.G[m + 1][0] = -Vn;
    o.Gb[m + 1][0] = v[m];
    o.G[m + 1][m + 1] = Vn;
    o.G[m + 1][a] = V[m];
    o.G[a][m + 1] = -bt_mul(k.c2, V[m]);
    o.G[4][m + 1] = o.G[a][m + 1];
    o.Gb[4][m + 1] = vn;
  }
  o.G[a][0] = fma(-Vn, vn, X);
  o.G[a][a] = k.two_m_c2;
  o.Gb[a][a] = Vn;
  o.G[a][4] = k.c2t2;
  o.G[4][0] = fma((T)2.0, X, -e1);
  o.Gb[4][0] = vn;
  o.G[4][a] = fma(-k.c2, Y, fma(-k.c2t2, q, e1));
  o.G[4][4] = k.c1;
  o.Gb[4][4] = Vn;
  const T kt = bt_mul(k.kc, ri), kn = bt_mul(k.k43, ri), g = bt_mul(k.kg, ri);
  const T wt = bt_add(kt, -g), wn = bt_add(kn, -g);
  o.H[0][0] = k.t1d[0];
  T s = bt_mul(g, E);
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const T km = m == DIR ? kn : kt;
    o.H[m + 1][0] = -bt_mul(km, v[m]);
    o.H[m + 1][m + 1] = fma(m == DIR ? k.k43 : k.kc, ri, k.t1d[m + 1]);
    o.H[4][m + 1] = bt_mul(m == DIR ? wn : wt, v[m]);
    s = fma(o.H[4][m + 1], v[m], s);
  }
  o.H[4][0] = -s;
  o.H[4][4] = fma(k.kg, ri, k.t1d[4]);
}

template <int DIR, typename T>
__device__ __forceinline__ void bt_form_p(const BtGH<DIR, T>& o, T P[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (anz<DIR>(r, c))
        P[r][c] = !hnz<DIR>(r, c)  ? o.G[r][c]
                  : !fnz<DIR>(r, c) ? o.H[r][c]
                  : gprod<DIR>(r, c) ? fma(o.G[r][c], o.Gb[r][c], o.H[r][c])
                                     : bt_add(o.G[r][c], o.H[r][c]);
}
template <int DIR, typename T>
__device__ __forceinline__ void bt_form_c(const BtGH<DIR, T>& o, T C[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (anz<DIR>(r, c))
        C[r][c] = !hnz<DIR>(r, c)  ? o.G[r][c]
                  : !fnz<DIR>(r, c) ? -o.H[r][c]
                  : gprod<DIR>(r, c) ? fma(o.G[r][c], o.Gb[r][c], -o.H[r][c])
                                     : bt_add(o.G[r][c], -o.H[r][c]);
}
template <int DIR, typename T>
__device__ __forceinline__ void bt_form_b(const BtGH<DIR, T>& o, T B[5][5]) {
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c)
      if (hnz<DIR>(r, c)) B[r][c] = r == c ? fma((T)2.0, o.H[r][c], (T)1.0) : (T)2.0 * o.H[r][c];
}

// Pivot reciprocal: FP64 by Newton-Raphson from the FP32 estimate (one ulp),
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
      if (bt_rank<D>(c) > s) B[p][c] = bt_mul(B[p][c], piv);
      if (bt_cset<D>(s, c)) C[p][c] = bt_mul(C[p][c], piv);
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
          C[q][c] = anz<D>(q, c) || (s > 0 && bt_cset<D>(s - 1, c)) ? fma(-m, C[p][c], C[q][c]) : -bt_mul(m, C[p][c]);
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
        C[q][c] = s < 4 || bt_cset<DIR>(bt_rank<DIR>(q), c) ? fma(-m, C[p][c], C[q][c]) : -bt_mul(m, C[p][c]);
      r[q] = fma(-m, r[p], r[q]);
    }
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

// State of one point: 1/rho and q from compute_rhs's primitive planes, momenta
// and energy from u as it is at the call, as the reference's sweeps take them.
// The velocities are formed where the state is used, not where it is loaded
// ahead (the products wait for the loads); they are the velocity planes' bits
// while u is the u of those planes.
template <typename T>
struct BtState {
  T ri, u[4], q;
};
template <typename T>
__device__ __forceinline__ BtState<T> bt_load_state(const Fields& F, int64_t pt) {
  const int64_t NP = F.NP;
  BtState<T> s;
  s.ri = (T)F.prim[PR_RHOI * NP + pt];
#pragma unroll
  for (int m = 0; m < 4; ++m) s.u[m] = (T)F.u[(m + 1) * NP + pt];
  s.q = (T)F.prim[PR_QS * NP + pt];
  return s;
}
template <int DIR, typename T>
__device__ __forceinline__ void bt_gh(const BtK<T>& k, const BtState<T>& s, BtGH<DIR, T>& o) {
  const T v[3] = {bt_mul(s.u[0], s.ri), bt_mul(s.u[1], s.ri), bt_mul(s.u[2], s.ri)};
  bt_gh<DIR, T>(k, s.ri, v, bt_mul(s.u[3], s.ri), s.q, o);
}

// The line solve, one thread per line (src/BT/x_solve.jl:444-488,501-1746 and
// its y, z copies): C'_p goes to the line scratch lhsc[(p*25 + e) * nlt +
// line], the eliminated rhs back into rhs.  The next point's state and rhs
// are loaded one step ahead.
template <int DIR, typename T>
__device__ __forceinline__ void bt_line_item(const Fields& F, const Consts& K, const Work w, T* __restrict__ lhsc,
                                             int64_t nlt, int add_u) {
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
  T rp[5], Cp[5][5], Pcur[5][5], Pnext[5][5], Bs[5][5];
  BtGH<DIR, T> J;
  BtState<T> s = bt_load_state<T>(F, base);
  bt_gh<DIR, T>(k, s, J);
  bt_form_p<DIR, T>(J, Pcur);
  s = bt_load_state<T>(F, base + st);
  bt_gh<DIR, T>(k, s, J);
  bt_form_p<DIR, T>(J, Pnext);
  bt_form_b<DIR, T>(J, Bs);
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
    bt_gh<DIR, T>(k, sp, J);
    bt_form_c<DIR, T>(J, C);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b)
        if (anz<DIR>(a, b)) Pcur[a][b] = Pnext[a][b];
    bt_form_p<DIR, T>(J, Pnext);
    bt_form_b<DIR, T>(J, Bs);
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

template <int DIR, typename T>
__global__ void __launch_bounds__(128) k_bt_line(Fields F, Consts K, const Work* __restrict__ work, int nwork,
                                                 T* __restrict__ lhsc, int64_t nlt, int add_u) {
  for (int it = blockIdx.x; it < nwork; it += gridDim.x) bt_line_item<DIR, T>(F, K, work[it], lhsc, nlt, add_u);
}

// ---------------------------------------------------------------------------
// The same solve for launches with too few lines to give every SM quarter a
// warp (FP64): twelve lanes per line, five lines per block of two warps.  An
// SM quarter takes an FP64 warp instruction every 64 cycles whatever its
// active lanes, and a line advances one point per 300 or so instructions of
// k_bt_line; here its work is spread over lanes and over both its ends.
//   - Warp 0 eliminates each line from point 0 up to the middle, warp 1 from
//     point n-1 down (the same line with G turned to -G).  At the seam
//     x_A = r'_A - C'_A x_B and x_B = r'_B - C'_B x_A, so each half solves
//     (I - C'_A C'_B) x_A = r'_A - C'_A r'_B and substitutes back to its end.
//   - G, H, P, B, C of six consecutive points at a time, one point per lane,
//     into shared memory (they do not depend on the elimination).
//   - Lane c < 5 keeps column c of C', lane 5 keeps r': B' and r' are one
//     column per lane (18 multiply-adds), and each step of the elimination
//     takes the pivot column from its lane by shuffles and updates the lane's
//     column of B' and its column of C (lane 5: r'), about 95 instructions per
//     lane and point.
//   - Back substitution: lane i < 5 holds row i.
// ADJ: the transposed system of the adjoint (rows 0..n-1 of T^T, all blocks of
// row p from the Jacobian at p): -C^T, B^T and -P^T in the places of P, B and
// C, identity rows at the ends, r the adjoint in place.
// Sweeps in us, k_bt_line / six lanes from one end / here: 24x24x6 x and y
// 217 / 74 / 45, z 65 / 25 / 20; 64x64x8 362 / 120 / 81, z (8 points) 95 / 39 /
// 52; 128x128x16 x 746 / 383 / 340 (few_lines in npbmz_api.cu draws the line).
// ---------------------------------------------------------------------------
constexpr int BTS_LINES = 5;   // lines per block
constexpr int BTS_LANES = 6;   // lanes per half of a line
constexpr int BTS_PTS = 6;     // points assembled at a time
constexpr int BTS_SLOTS = 8;   // points kept: a block of points and the two before it
constexpr int BTS_E = 18 + 25 + 25 + 5;  // doubles per point: P (nonzeros), B, C, rhs
constexpr int BTS_RING = BTS_SLOTS * BTS_E * BTS_LINES;  // doubles per warp
constexpr size_t BTS_SMEM = (size_t)(2 * BTS_RING + 2 * BTS_LINES * 30) * sizeof(double);
static_assert(BTS_SMEM <= 48 * 1024, "no opt-in to larger shared memory");

template <int DIR>
__host__ __device__ constexpr int bt_pidx(int r, int c) {  // place of P's entry (r, c) among its 18 nonzeros
  int n = 0;
  for (int rr = 0; rr < 5; ++rr)
    for (int cc = 0; cc < 5; ++cc) {
      if (rr == r && cc == c) return n;
      if (anz<DIR>(rr, cc)) ++n;
    }
  return n;
}

template <int DIR, bool ADJ>
__device__ __forceinline__ void bt_line12(const Fields& F, const Consts& K, const Work* __restrict__ work, int lpi,
                                          double* __restrict__ rhs, double* __restrict__ lhsc, int64_t nlt, int add_u,
                                          double* smem) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int half = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane < 30 ? lane / BTS_LANES : 0, c = lane < 30 ? lane - g * BTS_LANES : 5;
  const int off = blockIdx.y * BTS_LINES;
  const int last = min(w.first + lpi, zone_lines(Z, DIR)) - 1, want = w.first + off + g;
  if (w.first + off > last) return;  // the whole block
  const bool own = lane < 30 && want <= last;  // lanes without a line of their own compute line `last`, store nothing
  const int line = min(want, last);
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line, NP = F.NP;
  // rows first .. fin of this half, in its own index j: point j from its end
  const int rows = ADJ ? n : n - 2, near = (rows + 1) >> 1;
  const int first = ADJ ? 0 : 1, fin = first - 1 + (half ? rows - near : near);
  auto gq = [&](int j) -> int { return half ? n - 1 - j : j; };
  auto pnt = [&](int j) -> int64_t { return base + (int64_t)gq(j) * st; };
  BtK<double> k = bt_consts<double>(K, DIR);
  if (half) {
    k.t2 = -k.t2;
    k.c2t2 = -k.c2t2;
    k.c1t2 = -k.c1t2;
  }
  double* ring = smem + half * BTS_RING;
  auto at = [&](int j, int e) -> double& { return ring[((j % BTS_SLOTS) * BTS_E + e) * BTS_LINES + g]; };
  const unsigned all = 0xffffffffu;
  const int src0 = g * BTS_LANES;  // the group's lane 0
  const bool is_r = c == 5;
  const int col = is_r ? 0 : c;
  // this lane's point of the block of points j0 .. j0+5
  BtState<double> s;
  double fr[5];
  auto load = [&](int j0) {
    const int j = min(j0 + c, n - 1);
    s = bt_load_state<double>(F, pnt(j));
#pragma unroll
    for (int m = 0; m < 5; ++m) fr[m] = j <= fin || j == 0 ? rhs[m * NP + pnt(j)] : 0.0;
  };
  auto assemble = [&](int j0) {
    if (lane >= 30) return;
    BtGH<DIR, double> J;
    double M[5][5];
    const int j = j0 + c;
    const bool end = ADJ && (j == 0 || j >= n - 1);
    bt_gh<DIR, double>(k, s, J);
    bt_form_p<DIR, double>(J, M);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        if (ADJ) at(j, 43 + b * 5 + a) = anz<DIR>(a, b) && j <= n - 3 ? -M[a][b] : 0.0;
        else if (anz<DIR>(a, b)) at(j, bt_pidx<DIR>(a, b)) = M[a][b];
      }
    bt_form_b<DIR, double>(J, M);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b)
        at(j, 18 + (ADJ ? b * 5 + a : a * 5 + b)) = end ? (a == b ? 1.0 : 0.0) : hnz<DIR>(a, b) ? M[a][b] : 0.0;
    bt_form_c<DIR, double>(J, M);
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        if (!ADJ) at(j, 43 + a * 5 + b) = anz<DIR>(a, b) ? M[a][b] : 0.0;
        else if (anz<DIR>(a, b)) at(j, bt_pidx<DIR>(a, b)) = j >= 2 ? -M[a][b] : 0.0;
      }
#pragma unroll
    for (int m = 0; m < 5; ++m) at(j, 68 + m) = fr[m];
  };
  load(0);
  assemble(0);
  load(BTS_PTS);
  __syncwarp();
  double x[5];  // column c of C'_{j-1}, or r'_{j-1}
#pragma unroll
  for (int m = 0; m < 5; ++m) x[m] = is_r && !ADJ ? at(0, 68 + m) : 0.0;
  for (int j = first; j <= fin; ++j) {
    const int next = ADJ ? j : j + 1;  // the last point row j needs
    if (next > 0 && next % BTS_PTS == 0) {
      __syncwarp();  // the slots of the block before are free but its last two
      assemble(next);
      load(next + BTS_PTS);
      __syncwarp();
    }
    double b[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      b[i] = is_r ? at(j, 68 + i) : at(j, 18 + i * 5 + col);
#pragma unroll
      for (int e = 0; e < 5; ++e)
        if (anz<DIR>(ADJ ? e : i, ADJ ? i : e))
          b[i] = fma(at(ADJ ? j : j - 1, bt_pidx<DIR>(ADJ ? e : i, ADJ ? i : e)), x[e], b[i]);
    }
    // right-hand side column: C_j's, or r'
#pragma unroll
    for (int i = 0; i < 5; ++i) x[i] = is_r ? b[i] : at(next, 43 + i * 5 + col);
    double up[5][5];  // the pivot columns' entries above the diagonal, for the back step
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      const int pr = bt_piv<DIR>(t);
      double m[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        m[i] = __shfl_sync(all, b[i], src0 + pr);
        if (bt_rank<DIR>(i) < t) up[i][pr] = m[i];
      }
      const double piv = bt_recip(m[pr]);
      b[pr] *= piv;
      x[pr] *= piv;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        if (bt_rank<DIR>(i) <= t) continue;
        b[i] = fma(-m[i], b[pr], b[i]);
        x[i] = fma(-m[i], x[pr], x[i]);
      }
    }
#pragma unroll
    for (int t = 4; t > 0; --t) {
      const int pr = bt_piv<DIR>(t);
#pragma unroll
      for (int i = 0; i < 5; ++i)
        if (bt_rank<DIR>(i) < t) x[i] = fma(-up[i][pr], x[pr], x[i]);
    }
    if (own) {
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        if (is_r) rhs[i * NP + pnt(j)] = x[i];
        else lhsc[((int64_t)gq(j) * 25 + i * 5 + c) * nlt + gl] = x[i];
      }
    }
  }
  // the seam
  double* mine = smem + 2 * BTS_RING + (half * BTS_LINES + g) * 30;
  const double* other = smem + 2 * BTS_RING + ((1 - half) * BTS_LINES + g) * 30;
  if (lane < 30) {
#pragma unroll
    for (int i = 0; i < 5; ++i) mine[is_r ? 25 + i : i * 5 + c] = x[i];
  }
  __syncthreads();
  double y;  // row `row` of the solution at row fin
  const int row = col;
  {
    double b[5], up[5][5];
#pragma unroll
    for (int i = 0; i < 5; ++i) b[i] = is_r ? x[i] : i == c ? 1.0 : 0.0;
#pragma unroll
    for (int e = 0; e < 5; ++e) {
      const double v = is_r ? other[25 + e] : other[e * 5 + col];
#pragma unroll
      for (int i = 0; i < 5; ++i) b[i] = fma(-mine[i * 5 + e], v, b[i]);
    }
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      double m[5];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        m[i] = __shfl_sync(all, b[i], src0 + t);
        if (i < t) up[i][t] = m[i];
      }
      b[t] *= bt_recip(m[t]);
#pragma unroll
      for (int i = t + 1; i < 5; ++i) b[i] = fma(-m[i], b[t], b[i]);
    }
#pragma unroll
    for (int t = 4; t > 0; --t)
#pragma unroll
      for (int i = 0; i < t; ++i) b[i] = fma(-up[i][t], b[t], b[i]);
    y = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const double v = __shfl_sync(all, b[i], src0 + 5);
      if (row == i) y = v;
    }
  }
  // back substitution by rows; row c of C'_j and r'_j are loaded BACK steps ahead
  constexpr int BACK = 4;
  double cq[BACK][5], rq[BACK], uq[BACK];
  auto fetch = [&](int j, int slot) {
    if (j < first) return;
#pragma unroll
    for (int e = 0; e < 5; ++e) cq[slot][e] = lhsc[((int64_t)gq(j) * 25 + row * 5 + e) * nlt + gl];
    rq[slot] = rhs[row * NP + pnt(j)];
    uq[slot] = add_u ? F.u[row * NP + pnt(j)] : 0.0;
  };
  auto store = [&](int j, double uv) {
    if (!own || is_r) return;
    rhs[row * NP + pnt(j)] = y;
    if (add_u) F.u[row * NP + pnt(j)] = uv + y;
  };
#pragma unroll
  for (int q = 0; q < BACK; ++q) fetch(fin - 1 - q, q);
  if (fin >= first) store(fin, add_u ? F.u[row * NP + pnt(fin)] : 0.0);
  for (int j0 = fin - 1; j0 >= first; j0 -= BACK) {
#pragma unroll
    for (int q = 0; q < BACK; ++q) {
      const int j = j0 - q;
      if (j < first) break;
      double t = rq[q];
#pragma unroll
      for (int e = 0; e < 5; ++e) t = fma(-cq[q][e], __shfl_sync(all, y, src0 + e), t);
      y = t;
      store(j, uq[q]);
      fetch(j - BACK, q);
    }
  }
}

template <int DIR>
__global__ void __launch_bounds__(64, 1) k_bt_line12(Fields F, Consts K, const Work* __restrict__ work, int lpi,
                                                     double* __restrict__ lhsc, int64_t nlt, int add_u) {
  extern __shared__ double bts[];
  bt_line12<DIR, false>(F, K, work, lpi, F.rhs, lhsc, nlt, add_u, bts);
}
