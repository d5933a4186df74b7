// quad.cuh -- quadrature pieces of the element actions y_K = A_K x_K.
//
// In barycentric coordinates, with g_a = grad(lambda_a):
//   P2 basis derivatives  dphi_v/dl_a = delta_va (4 l_v - 1),
//                         dphi_(p,q)/dl_p = 4 l_q, dphi_(p,q)/dl_q = 4 l_p;
//   grad u = sum_a U_a g_a,  U_a = sum_j x_j dphi_j/dl_a;
//   y_j  += w |T| sum_a dphi_j/dl_a S_a,  S_a = flux . g_a,
// where the flux is kappa grad u (diffusion) or the stress row
// sigma_c = lambda div(u) e_c + mu (grad u + grad u^T)_c (elasticity, output
// component c).  The rules integrate the element integrands exactly: P1 -- the
// centroid (kappa linear, gradients constant); P2 diffusion -- degree 3 (kappa
// linear times two linear gradients); P2 elasticity -- degree 2.
#pragma once

#include "assemble.cuh"

namespace db2 {
namespace dev {

template <int D, int DEG>
struct Quad;
template <int D>
struct Quad<D, 1> {  // centroid
  static constexpr int NQ = 1;
  __host__ __device__ static constexpr double w(int) { return 1.0; }
  __host__ __device__ static constexpr double lam(int, int) { return 1.0 / (D + 1); }
};
// Hammer-Marlowe-Stroud tetrahedron rule of degree 2: (a, b, b, b) and
// permutations, a = (5 + 3 sqrt 5) / 20, b = (5 - sqrt 5) / 20, weights 1/4.
template <>
struct Quad<3, 2> {
  static constexpr int NQ = 4;
  __host__ __device__ static constexpr double w(int) { return 0.25; }
  __host__ __device__ static constexpr double lam(int q, int a) {
    return a == q ? 0.5854101966249685 : 0.1381966011250105;
  }
};
// Stroud's degree-3 rules: tetrahedron -4/5 at the centroid and 9/20 at
// (1/2, 1/6, 1/6, 1/6) and permutations; triangle -27/48 at the centroid and
// 25/48 at (3/5, 1/5, 1/5) and permutations.
template <>
struct Quad<3, 3> {
  static constexpr int NQ = 5;
  __host__ __device__ static constexpr double w(int q) { return q == 0 ? -0.8 : 0.45; }
  __host__ __device__ static constexpr double lam(int q, int a) {
    return q == 0 ? 0.25 : (a == q - 1 ? 0.5 : 1.0 / 6.0);
  }
};
template <>
struct Quad<2, 3> {
  static constexpr int NQ = 4;
  __host__ __device__ static constexpr double w(int q) { return q == 0 ? -27.0 / 48.0 : 25.0 / 48.0; }
  __host__ __device__ static constexpr double lam(int q, int a) {
    return q == 0 ? 1.0 / 3.0 : (a == q - 1 ? 0.6 : 0.2);
  }
};

// grad(lambda_a) of the affine simplex and |T|.
template <int D>
__device__ __forceinline__ double bary_gradients(const double (&x)[D + 1][D], double (&g)[D + 1][D]) {
  Geometry<D> G;
  geometry(x, G);  // n[a] = det(J) grad(lambda_a), vol = |T|
  double det;
  if constexpr (D == 3) {
    det = (x[1][0] - x[0][0]) * G.n[1][0] + (x[1][1] - x[0][1]) * G.n[1][1] + (x[1][2] - x[0][2]) * G.n[1][2];
  } else {
    det = (x[1][0] - x[0][0]) * G.n[1][0] + (x[1][1] - x[0][1]) * G.n[1][1];
  }
  // 1/det from the geometry's 1/(D! |det|)
  const double inv = (D == 3 ? 6.0 : 2.0) * G.s * (det < 0.0 ? -1.0 : 1.0);
#pragma unroll
  for (int a = 0; a <= D; ++a)
#pragma unroll
    for (int r = 0; r < D; ++r) g[a][r] = G.n[a][r] * inv;
  return G.vol;
}

// U_a = sum_j x_j dphi_j/dl_a at barycentric point l, for one component.
template <int D, int P, typename CT>
__device__ __forceinline__ CT node_derivative(const CT (&xc)[El<D, P>::K], const double (&l)[D + 1], int a) {
  constexpr int NB = D + 1;
  if constexpr (P == 1) {
    return xc[a];
  } else {
    CT u = CT(4.0 * l[a] - 1.0) * xc[a];
#pragma unroll
    for (int e = 0; e < El<D, P>::NE; ++e) {
      const int p0 = edge_end(D, e, 0), p1 = edge_end(D, e, 1);
      if (p0 == a) u = fma(CT(4.0 * l[p1]), xc[NB + e], u);
      if (p1 == a) u = fma(CT(4.0 * l[p0]), xc[NB + e], u);
    }
    return u;
  }
}

// y_j += sum_a dphi_j/dl_a S_a at barycentric point l.
template <int D, int P, typename CT>
__device__ __forceinline__ void test_basis(const CT (&S)[D + 1], const double (&l)[D + 1],
                                           double (&y)[El<D, P>::K]) {
  constexpr int NB = D + 1;
#pragma unroll
  for (int v = 0; v < NB; ++v) y[v] += double(P == 1 ? S[v] : CT(4.0 * l[v] - 1.0) * S[v]);
  if constexpr (P == 2) {
#pragma unroll
    for (int e = 0; e < El<D, P>::NE; ++e) {
      const int p0 = edge_end(D, e, 0), p1 = edge_end(D, e, 1);
      y[NB + e] += double(fma(CT(4.0 * l[p1]), S[p0], CT(4.0 * l[p0]) * S[p1]));
    }
  }
}

}  // namespace dev
}  // namespace db2
