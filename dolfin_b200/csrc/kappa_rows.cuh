// kappa_rows.cuh -- FP64 element-matrix rows of kappa*grad(u).grad(v) with a P1
// kappa on quadratic simplices, with few operations.
//
// The generated rows (generated/element_rows.h) expand every coefficient of the
// geometry tensor in the kappa values.  By moments they have a common form:
// with S = sum kappa, int kappa lambda_i lambda_m is, in units of |T| D!/(D+3)!,
// K_im = S + kappa_i + kappa_m (i != m) and K_ii = 2 S + 4 kappa_i.  For the row
// of the edge (0, 1), with u = S + kappa_0, w = S + kappa_1 and the geometry
// tensor W_ab = |T| g_a.g_b, the entries are
//   vertex v:    W_0v (4 K_1v - (D+3) w) + W_1v (4 K_0v - (D+3) u)
//   edge (p,q):  4 (W_0p K_1q + W_0q K_1p + W_1p K_0q + W_1q K_0p),
// and for the row of vertex 0, with c_m = 4 K_0m - (D+3) (S + kappa_m),
//   vertex v:    W_0v (4 c_v - sum c) / 4
//   edge (p,q):  W_0p c_q + W_0q c_p
// (both up to the scales that the callers fold into W: the generated rows').
// Edge row of a tetrahedron: 23 operations for the coefficients against 43,
// vertex row 15 against 42, of about 165 and 110 a cell and row in all.
#pragma once

namespace db2 {
namespace dev {

// Local edges after the vertices: (2,3)(1,3)(1,2)(0,3)(0,2)(0,1) and
// (1,2)(0,2)(0,1).
__device__ __forceinline__ void p2_kappa_edge_row(const double (&W)[2][4], const double (&k)[4], double (&o)[10]) {
  const double S = (k[0] + k[1]) + (k[2] + k[3]);
  const double u = S + k[0], w = S + k[1];
  const double u2 = 2.0 * u, w2 = 2.0 * w;
  // P_m = 2 K_1m, R_m = 2 K_0m
  const double R1 = fma(2.0, k[1], u2), R2 = fma(2.0, k[2], u2), R3 = fma(2.0, k[3], u2);
  const double P2 = fma(2.0, k[2], w2), P3 = fma(2.0, k[3], w2);
  const double R0 = fma(2.0, u2, 4.0 * k[0]), P1 = fma(2.0, w2, 4.0 * k[1]);
  o[0] = fma(W[1][0], fma(4.0, k[0], u), W[0][0] * fma(2.0, k[0], -w));
  o[1] = fma(W[1][1], fma(2.0, k[1], -u), W[0][1] * fma(4.0, k[1], w));
  o[2] = fma(W[1][2], fma(2.0, k[2], -u), W[0][2] * fma(2.0, k[2], -w));
  o[3] = fma(W[1][3], fma(2.0, k[3], -u), W[0][3] * fma(2.0, k[3], -w));
  o[4] = fma(W[1][3], R2, fma(W[1][2], R3, fma(W[0][3], P2, W[0][2] * P3)));
  o[5] = fma(W[1][3], R1, fma(W[1][1], R3, fma(W[0][3], P1, W[0][1] * P3)));
  o[6] = fma(W[1][2], R1, fma(W[1][1], R2, fma(W[0][2], P1, W[0][1] * P2)));
  o[7] = fma(W[1][3], R0, fma(W[1][0], R3, fma(W[0][3], R1, W[0][0] * P3)));
  o[8] = fma(W[1][2], R0, fma(W[1][0], R2, fma(W[0][2], R1, W[0][0] * P2)));
  o[9] = fma(W[1][1], R0, fma(W[1][0] + W[0][1], R1, W[0][0] * P1));
}
__device__ __forceinline__ void p2_kappa_vertex_row(const double (&W)[1][4], const double (&k)[4], double (&o)[10]) {
  const double S = (k[0] + k[1]) + (k[2] + k[3]);
  const double S4 = 4.0 * S;
  const double c0 = fma(20.0, k[0], S4), h = fma(8.0, k[0], -S4), v = fma(-4.0, k[0], -S);
  const double c1 = fma(-4.0, k[1], h), c2 = fma(-4.0, k[2], h), c3 = fma(-4.0, k[3], h);
  o[0] = W[0][0] * fma(7.0, S, 8.0 * k[0]);
  o[1] = W[0][1] * fma(-4.0, k[1], v);
  o[2] = W[0][2] * fma(-4.0, k[2], v);
  o[3] = W[0][3] * fma(-4.0, k[3], v);
  o[4] = fma(W[0][3], c2, W[0][2] * c3);
  o[5] = fma(W[0][3], c1, W[0][1] * c3);
  o[6] = fma(W[0][2], c1, W[0][1] * c2);
  o[7] = fma(W[0][3], c0, W[0][0] * c3);
  o[8] = fma(W[0][2], c0, W[0][0] * c2);
  o[9] = fma(W[0][1], c0, W[0][0] * c1);
}
__device__ __forceinline__ void p2_kappa_edge_row(const double (&W)[2][3], const double (&k)[3], double (&o)[6]) {
  const double S = (k[0] + k[1]) + k[2];
  const double u = S + k[0], w = S + k[1];
  const double u4 = 4.0 * u, w4 = 4.0 * w;
  // P_m = 4 K_1m, R_m = 4 K_0m
  const double R1 = fma(4.0, k[1], u4), R2 = fma(4.0, k[2], u4), P2 = fma(4.0, k[2], w4);
  const double R0 = fma(2.0, u4, 8.0 * k[0]), P1 = fma(2.0, w4, 8.0 * k[1]);
  o[0] = fma(W[1][0], fma(3.0, u, 8.0 * k[0]), W[0][0] * fma(4.0, k[0], -w));
  o[1] = fma(W[1][1], fma(4.0, k[1], -u), W[0][1] * fma(3.0, w, 8.0 * k[1]));
  o[2] = fma(W[1][2], fma(4.0, k[2], -u), W[0][2] * fma(4.0, k[2], -w));
  o[3] = fma(W[1][2], R1, fma(W[1][1], R2, fma(W[0][2], P1, W[0][1] * P2)));
  o[4] = fma(W[1][2], R0, fma(W[1][0], R2, fma(W[0][2], R1, W[0][0] * P2)));
  o[5] = fma(W[1][1], R0, fma(W[1][0] + W[0][1], R1, W[0][0] * P1));
}
__device__ __forceinline__ void p2_kappa_vertex_row(const double (&W)[1][3], const double (&k)[3], double (&o)[6]) {
  const double S = (k[0] + k[1]) + k[2];
  const double S3 = 3.0 * S;
  const double c0 = fma(11.0, k[0], S3), h = fma(4.0, k[0], -S), v = S + k[0];
  const double c1 = h - k[1], c2 = h - k[2];
  o[0] = W[0][0] * fma(6.0, k[0], S3);
  o[1] = W[0][1] * (-v - k[1]);
  o[2] = W[0][2] * (-v - k[2]);
  o[3] = fma(W[0][2], c1, W[0][1] * c2);
  o[4] = fma(W[0][2], c0, W[0][0] * c2);
  o[5] = fma(W[0][1], c0, W[0][0] * c1);
}

}  // namespace dev
}  // namespace db2
