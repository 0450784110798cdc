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
// they fill.  Every multiply-add is written as fma, so that the two mappings
// of the FP64 solve (one thread per line, six lanes per line) give the same
// bits.  One point takes 389 FP64 instructions (531 with the blocks
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
  T rp[5], Cp[5][5], Pcur[5][5], Pnext[5][5], Bs[5][5];
  BtGH<DIR, T> J;
  BtState<T> s = bt_load_state<T>(F, base);
  bt_gh<DIR, T>(k, s.ri, s.v, s.u5 * s.ri, s.q, J);
  bt_form_p<DIR, T>(J, Pcur);
  s = bt_load_state<T>(F, base + st);
  bt_gh<DIR, T>(k, s.ri, s.v, s.u5 * s.ri, s.q, J);
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
    bt_gh<DIR, T>(k, sp.ri, sp.v, sp.u5 * sp.ri, sp.q, J);
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

// ---------------------------------------------------------------------------
// The same solve with six lanes per line (FP64), five lines per warp, one
// warp per block: for launches with too few lines to give every SM quarter a
// warp.  An SM quarter takes an FP64 warp instruction every 64 cycles
// whatever its active lanes, and a line advances one point per 389
// instructions of k_bt_line; here the work of a point is spread over the
// group's lanes, about 95 instructions per lane (and 1.6 times k_bt_line's
// warp instructions in all, so full launches keep that one).  Sweeps (us,
// k_bt_line / here): 24x24x6 x and y 217 / 74, z 65 / 25; 64x64x8 362 / 120,
// 95 / 39; 128x128x16 746 / 381, z 235 / 303; 304x208x17 x 1123 / 1177, z
// 653 / 1105 (few_lines in npbmz_api.cu draws the line).
//   - G, H, P, B, C of six consecutive points at a time, one point per lane,
//     into shared memory (they do not depend on the elimination);
//   - lane c < 5 keeps column c of C', lane 5 keeps r': B' and r' are one
//     column per lane (18 multiply-adds), and each step of the elimination
//     takes the pivot column from its lane by shuffles and updates the lane's
//     column of B' and its column of C (lane 5: r');
//   - back substitution: lane i < 5 holds row i.
// Each element sees the operations of k_bt_line in the same order (those
// k_bt_line skips multiply structural zeros), so the results are the same.
// ---------------------------------------------------------------------------
constexpr int BTS_LINES = 5;   // lines per warp
constexpr int BTS_LANES = 6;   // lanes per line
constexpr int BTS_PTS = 6;     // points assembled at a time
constexpr int BTS_E = 18 + 25 + 25 + 5;  // doubles per point: P (nonzeros), B, C, rhs
constexpr size_t BTS_SMEM = (size_t)2 * BTS_PTS * BTS_E * BTS_LINES * sizeof(double);

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

// ADJ: the transposed system of the adjoint instead (rows 0..n-1 of T^T, all
// blocks of row p from the Jacobian at p): -C^T, B^T and -P^T in the places of
// P, B and C, identity rows at the ends, r the adjoint in place.
template <int DIR, bool ADJ>
__device__ __forceinline__ void bt_line6(const Fields& F, const Consts& K, const Work* __restrict__ work, int lpi,
                                         double* __restrict__ rhs, double* __restrict__ lhsc, int64_t nlt, int add_u,
                                         double* bts) {
  const Work w = work[blockIdx.x];
  const ZoneDev Z = F.zones[w.zone];
  const int lane = threadIdx.x, g = lane < 30 ? lane / BTS_LANES : 0, c = lane < 30 ? lane - g * BTS_LANES : 5;
  const int off = blockIdx.y * BTS_LINES;
  const int last = min(w.first + lpi, zone_lines(Z, DIR)) - 1, want = w.first + off + g;
  if (w.first + off > last) return;  // the whole warp
  const bool own = lane < 30 && want <= last;  // lanes without a line of their own compute line `last`, store nothing
  const int line = min(want, last);
  int64_t base, st;
  line_geometry(Z, DIR, line, base, st);
  const int n = zone_line_len(Z, DIR);
  const int64_t gl = Z.lineoff[DIR] + line, NP = F.NP;
  const BtK<double>& k = bt_consts<double>(K, DIR);
  auto at = [&](int q, int e) -> double& { return bts[((q % (2 * BTS_PTS)) * BTS_E + e) * BTS_LINES + g]; };
  const unsigned all = 0xffffffffu;
  const int src0 = g * BTS_LANES;  // the group's lane 0
  // this lane's point of the block of points q0 .. q0+5
  BtState<double> s;
  double fr[5];
  auto load = [&](int q0) {
    const int q = min(q0 + c, n - 1);
    s = bt_load_state<double>(F, base + (int64_t)q * st);
#pragma unroll
    for (int m = 0; m < 5; ++m) fr[m] = rhs[m * NP + base + (int64_t)q * st];
  };
  auto assemble = [&](int q0) {
    if (lane >= 30) return;
    BtGH<DIR, double> J;
    double M[5][5];
    const int q = q0 + c;
    bt_gh<DIR, double>(k, s.ri, s.v, s.u5 * s.ri, s.q, J);
    const bool end = ADJ && (q == 0 || q >= n - 1);
    bt_form_p<DIR, double>(J, M);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        if (ADJ) at(q, 43 + j * 5 + i) = anz<DIR>(i, j) && q <= n - 3 ? -M[i][j] : 0.0;
        else if (anz<DIR>(i, j)) at(q, bt_pidx<DIR>(i, j)) = M[i][j];
      }
    bt_form_b<DIR, double>(J, M);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j)
        at(q, 18 + (ADJ ? j * 5 + i : i * 5 + j)) = end ? (i == j ? 1.0 : 0.0) : hnz<DIR>(i, j) ? M[i][j] : 0.0;
    bt_form_c<DIR, double>(J, M);
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        if (!ADJ) at(q, 43 + i * 5 + j) = anz<DIR>(i, j) ? M[i][j] : 0.0;
        else if (anz<DIR>(i, j)) at(q, bt_pidx<DIR>(i, j)) = q >= 2 ? -M[i][j] : 0.0;
      }
#pragma unroll
    for (int m = 0; m < 5; ++m) at(q, 68 + m) = fr[m];
  };
  const bool is_r = c == 5;
  const int col = is_r ? 0 : c;
  load(0);
  assemble(0);
  load(BTS_PTS);
  __syncwarp();
  double x[5];  // column c of C'_{p-1}, or r'_{p-1}
#pragma unroll
  for (int m = 0; m < 5; ++m) x[m] = is_r && !ADJ ? at(0, 68 + m) : 0.0;
  const int first = ADJ ? 0 : 1, fin = ADJ ? n - 1 : n - 2;
  for (int p = first; p <= fin; ++p) {
    const int last_q = ADJ ? p : p + 1;  // the last point row p needs
    if (last_q > 0 && last_q % BTS_PTS == 0) {
      __syncwarp();  // the slots of the block before the last are free
      assemble(last_q);
      load(last_q + BTS_PTS);
      __syncwarp();
    }
    double b[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      b[i] = is_r ? at(p, 68 + i) : at(p, 18 + i * 5 + col);
#pragma unroll
      for (int e = 0; e < 5; ++e)
        if (anz<DIR>(ADJ ? e : i, ADJ ? i : e))
          b[i] = fma(at(ADJ ? p : p - 1, bt_pidx<DIR>(ADJ ? e : i, ADJ ? i : e)), x[e], b[i]);
    }
    // right-hand side column: C_p's, or r'
#pragma unroll
    for (int i = 0; i < 5; ++i) x[i] = is_r ? b[i] : at(last_q, 43 + i * 5 + col);
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
      const int64_t pt = base + (int64_t)p * st;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        if (is_r) rhs[i * NP + pt] = x[i];
        else lhsc[((int64_t)p * 25 + i * 5 + c) * nlt + gl] = x[i];
      }
    }
  }
  // back substitution by rows; row c of C'_p and r'_p are loaded BACK steps ahead
  __syncwarp();
  constexpr int BACK = 4;
  const int row = col;
  double cq[BACK][5], rq[BACK], uq[BACK];
  auto fetch = [&](int p, int slot) {
    if (p < first) return;
    const int64_t pt = base + (int64_t)p * st;
#pragma unroll
    for (int e = 0; e < 5; ++e) cq[slot][e] = lhsc[((int64_t)p * 25 + row * 5 + e) * nlt + gl];
    rq[slot] = rhs[row * NP + pt];
    uq[slot] = add_u ? F.u[row * NP + pt] : 0.0;
  };
  double y = ADJ ? 0.0 : rhs[row * NP + base + (int64_t)(n - 1) * st];
#pragma unroll
  for (int q = 0; q < BACK; ++q) fetch(fin - q, q);
  for (int p0 = fin; p0 >= first; p0 -= BACK) {
#pragma unroll
    for (int q = 0; q < BACK; ++q) {
      const int p = p0 - q;
      if (p < first) break;
      double t = rq[q];
#pragma unroll
      for (int e = 0; e < 5; ++e) t = fma(-cq[q][e], __shfl_sync(all, y, src0 + e), t);
      y = t;
      if (own && !is_r) {
        const int64_t pt = base + (int64_t)p * st;
        rhs[row * NP + pt] = y;
        if (add_u) F.u[row * NP + pt] = uq[q] + y;
      }
      fetch(p - BACK, q);
    }
  }
}

template <int DIR>
__global__ void __launch_bounds__(32, 1) k_bt_line6(Fields F, Consts K, const Work* __restrict__ work, int lpi,
                                                    double* __restrict__ lhsc, int64_t nlt, int add_u) {
  extern __shared__ double bts[];
  bt_line6<DIR, false>(F, K, work, lpi, F.rhs, lhsc, nlt, add_u, bts);
}
