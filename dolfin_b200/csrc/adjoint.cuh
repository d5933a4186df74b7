// adjoint.cuh -- the adjoint dL/dkappa of one cell, by its local nodes.
#pragma once

#include <utility>

#include "assemble.cuh"

namespace db2 {
namespace dev {

// Quadratic elements in FP64: the row's part by moments (kappa_rows.cuh).  An
// entry is linear in K_0m and K_1m (edge row) or in c_m (vertex row), those in
// kappa; so the contraction with gA over the row's columns is taken first, per
// vertex m, and differentiated afterwards -- about 60 operations a row where
// contracting the row of every unit kappa takes 250.  W unscaled; t[k] is with
// respect to relabelled kappa_k, in units of |T| D!/(D+3)!.
template <int D>
__device__ __forceinline__ double p2_columns(const double (&W)[D + 1], const double (&g)[El<D, 2>::K], int m) {
  double a = g[m] * W[m];
#pragma unroll
  for (int p = 0; p <= D; ++p)
    if (p != m) a = fma(g[D + 1 + cell_edge_of(D, p, m)], W[p], a);
  return a;
}
template <int D>
__device__ __forceinline__ void vjp_edge_row(const double (&W0)[D + 1], const double (&W1)[D + 1],
                                             const double (&g)[El<D, 2>::K], double (&t)[D + 1]) {
  double a[D + 1], b[D + 1], A = 0.0, B = 0.0, al = 0.0, be = 0.0;
#pragma unroll
  for (int m = 0; m <= D; ++m) {
    a[m] = p2_columns<D>(W0, g, m);
    b[m] = p2_columns<D>(W1, g, m);
    A += a[m];
    B += b[m];
    al = fma(g[m], W0[m], al);
    be = fma(g[m], W1[m], be);
  }
  const double all = fma(4.0, (A + a[1]) + (B + b[0]), -(D + 3.0) * (al + be));
#pragma unroll
  for (int k = 0; k <= D; ++k) {
    t[k] = fma(4.0, a[k] + b[k], all);
    if (k == 1) t[k] += fma(4.0, fma(2.0, a[1], A), -(D + 3.0) * al);
    if (k == 0) t[k] += fma(4.0, fma(2.0, b[0], B), -(D + 3.0) * be);
  }
#pragma unroll
  for (int k = 0; k <= D; ++k) t[k] *= 4.0;
}
template <int D>
__device__ __forceinline__ void vjp_vertex_row(const double (&W0)[D + 1], const double (&g)[El<D, 2>::K],
                                               double (&t)[D + 1]) {
  double h[D + 1], H = 0.0, ga = 0.0;
#pragma unroll
  for (int v = 0; v <= D; ++v) ga = fma(g[v], W0[v], ga);
#pragma unroll
  for (int m = 0; m <= D; ++m) {
    h[m] = fma(4.0, p2_columns<D>(W0, g, m), -ga);
    H += h[m];
  }
  const double all = fma(4.0, H + h[0], -(D + 3.0) * H);
#pragma unroll
  for (int k = 0; k <= D; ++k) {
    t[k] = fma(4.0 - (D + 3.0), h[k], all);
    if (k == 0) t[k] = fma(4.0, fma(2.0, h[0], H), t[k]);
  }
}

// The part of local node LI of the cell (a compile-time relabelling, so the
// permuted geometry tensor is register renaming):
// acc[a] += sum_j gA_(LI,j) dA^K_(LI,j)/dkappa_a + gb_LI db^K_LI/dkappa_a.
// Wn[a][b] = n_a . n_b in the cell's own vertex order; under the relabelling
// n'_a = +-n_perm[a], so W'_ab = Wn[perm[a]][perm[b]] (|det J| unchanged).
// row.get<LI>(g, gbi) gives gA at the row's relabelled local nodes and gb.
template <int D, int P, bool LOADK, typename CT, int LI, typename Row>
__device__ __forceinline__ void vjp_node(const AsmParams& p, const double (&Wn)[D + 1][D + 1], double s, double vol,
                                         const double (&fv)[D + 1], const Row& row, double (&acc)[D + 1]) {
  using E = El<D, P>;
  using R = Rows<D, P, CT>;
  constexpr int NB = D + 1;
  constexpr uint32_t code = perm_code(D, LI);
  constexpr bool vertex = LI <= D;
  double g[E::K], gbi = 0.0;
  row.template get<LI>(g, gbi);
  auto pm = [](int a) { return int((code >> (2 * a)) & 3u); };
  CT lk[NB];
  if constexpr (LOADK) {
    CT fc[NB];
#pragma unroll
    for (int a = 0; a < NB; ++a) fc[a] = CT(fv[pm(a)]);
    if constexpr (P == 2 && !vertex) R::e_kfp1(fc, lk);
    else R::v_kfp1(fc, lk);
  }
  if constexpr (P == 2 && sizeof(CT) == 8) {
    double W[2][NB], t[NB];
#pragma unroll
    for (int a = 0; a < (vertex ? 1 : 2); ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) W[a][b] = Wn[pm(a)][pm(b)];
    if constexpr (vertex) vjp_vertex_row<D>(W[0], g, t);
    else vjp_edge_row<D>(W[0], W[1], g, t);
    const double sc = s * p.kscale * (D == 3 ? 1.0 / 120 : 1.0 / 60);
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      double tm = t[m] * sc;
      if constexpr (LOADK) tm = fma(gbi, vol * lk[m] * p.fc[0], tm);
      acc[pm(m)] += tm;
    }
  } else {
  CT W0[1][NB];
  CT W1[2][NB];
  // W times the generated rows' scale (see element_rows.h)
  const double sv = s * (p.kscale * R::sv_kp1);
#pragma unroll
  for (int b = 0; b < NB; ++b) W0[0][b] = CT(Wn[pm(0)][pm(b)] * sv);
  if constexpr (P == 2) {
    const double se = s * (p.kscale * R::se_kp1);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) W1[a][b] = CT(Wn[pm(a)][pm(b)] * se);
  }
#pragma unroll
  for (int m = 0; m < NB; ++m) {
    CT unit[NB];
#pragma unroll
    for (int a = 0; a < NB; ++a) unit[a] = CT(a == m ? 1 : 0);
    CT d[E::K];
    if constexpr (P == 1 || vertex) R::v_kp1(W0, unit, d);
    else R::e_kp1(W1, unit, d);
    double t = 0.0;
#pragma unroll
    for (int j = 0; j < E::K; ++j) t = fma(g[j], double(d[j]), t);
    if constexpr (LOADK) t = fma(gbi, vol * double(lk[m]) * p.fc[0], t);
    // relabelled vertex m is original local vertex perm[m]
    acc[pm(m)] += t;
  }
  }
}

template <int D, int P, bool LOADK, typename CT, typename Row, int... LI>
__device__ __forceinline__ void vjp_nodes(const AsmParams& p, const double (&Wn)[D + 1][D + 1], double s, double vol,
                                          const double (&fv)[D + 1], const Row& row, double (&acc)[D + 1],
                                          std::integer_sequence<int, LI...>) {
  (vjp_node<D, P, LOADK, CT, LI>(p, Wn, s, vol, fv, row, acc), ...);
}

}  // namespace dev
}  // namespace db2
