// patch.cu -- matrix-free action y = A x over cell patches (PatchPlan): a CTA
// per patch stages its nodes' x and its vertices' coordinates in shared
// memory, a thread per cell computes the cell's action y_K = A_K x_K into
// shared memory, and the patch's nodes sum their cells there in ascending cell
// order.  Nodes shared between patches leave a partial sum per patch, added
// in patch order by a second kernel.  The order of additions is fixed, so the
// result is bitwise repeatable.
//
// Against writing every cell's action to HBM and gathering it per row (2 x 8
// bytes per cell and local node, 0.85 GB at P2 n=96), a patch moves its plan
// (60 B a cell), x, y and about one partial sum a cell.  Measured on B200, ms
// per action: vector P2 elasticity n=48 0.245 -> 0.087, P2 tets n=96 0.342 ->
// 0.230, P1 tets n=80 0.102 -> 0.060; with FP32 actions 63x70x57 0.084 ->
// 0.079 (its quadrature is unchanged, and issue-bound).  Least is gained where
// the cell actions were short: P1 triangles with a constant coefficient in FP32
// take 0.0165 against 0.0142 at n=600, 0.0226 / 0.0257 at n=900, 0.0637 / 0.0618
// at n=1500, 0.101 / 0.105 at n=2000.
#include <cuda_runtime.h>

#include "patch.cuh"
#include "quad.cuh"

namespace db2 {
namespace dev {

struct PatchArgs : PatchView {
  const double* xw;     // vertex records, coordinates first
  const double* kappa;  // P1 field or null
  double kscale, mu, lmbda;
  const double* x;
  double* y;
  int64_t nnodes;
};

// Element action of P2 by exact moments.  With U_m the gradient of u at
// vertex m (grad u is linear), F the flux and M_m = int lambda_m F:
//   y_v = g_v . (4 M_v - sum_m M_m),   y_(p,q) = 4 (g_p . M_q + g_q . M_p),
// where for a linear flux (F_m its vertex values) M_m = |T| c2 (sum F + F_m),
// and for F = kappa grad u with linear kappa, by int lambda_m lambda_k lambda_l,
//   M_m = |T| c3 [(sum kappa)(sum U) + sum kappa_k U_k + kappa_m (sum U + 2 U_m)
//                 + (sum kappa) U_m].
// About half the operations of the quadrature of the same degree (P2
// tetrahedra, linear kappa: ~230 against ~430).
template <int D>
constexpr double moment2() { return D == 3 ? 1.0 / 20 : 1.0 / 12; }
template <int D>
constexpr double moment3() { return D == 3 ? 1.0 / 120 : 1.0 / 60; }

// Gradients of one P2 component at the vertices: U_m = sum_a d_a g_a with
// d_a = 4 x_(a,m) - x_a (a != m), 3 x_m (a = m).
template <int D, typename CT>
__device__ __forceinline__ void p2_vertex_gradients(const CT (&xc)[El<D, 2>::K], const CT (&g)[D + 1][D],
                                                    CT (&U)[D + 1][D]) {
#pragma unroll
  for (int m = 0; m <= D; ++m) {
#pragma unroll
    for (int r = 0; r < D; ++r) U[m][r] = CT(0);
#pragma unroll
    for (int a = 0; a <= D; ++a) {
      const CT d = a == m ? CT(3) * xc[m] : fma(CT(4), xc[D + 1 + cell_edge_of(D, a, m)], -xc[a]);
#pragma unroll
      for (int r = 0; r < D; ++r) U[m][r] = fma(d, g[a][r], U[m][r]);
    }
  }
}

template <int D, typename CT>
__device__ __forceinline__ CT dotg(const CT (&a)[D], const CT (&b)[D]) {
  CT s = a[0] * b[0];
#pragma unroll
  for (int r = 1; r < D; ++r) s = fma(a[r], b[r], s);
  return s;
}

// P2 test functions against the moments M and t_v = 4 M_v - sum M.
template <int D, typename CT>
__device__ __forceinline__ void p2_test(const CT (&M)[D + 1][D], const CT (&t)[D + 1][D], const CT (&g)[D + 1][D],
                                        CT (&y)[El<D, 2>::K]) {
#pragma unroll
  for (int v = 0; v <= D; ++v) y[v] = dotg<D, CT>(g[v], t[v]);
#pragma unroll
  for (int e = 0; e < El<D, 2>::NE; ++e) {
    const int p = edge_end(D, e, 0), q = edge_end(D, e, 1);
    CT s = dotg<D, CT>(g[p], M[q]);
#pragma unroll
    for (int r = 0; r < D; ++r) s = fma(g[q][r], M[p][r], s);
    y[D + 1 + e] = CT(4) * s;
  }
}

// A linear flux of vertex values F: M_m = S + F_m with S = sum F (times |T|
// c2), so t_v = 4 F_v - (D - 2) S.
template <int D, typename CT>
__device__ __forceinline__ void p2_test_linear(const CT (&F)[D + 1][D], const CT (&g)[D + 1][D],
                                               CT (&y)[El<D, 2>::K]) {
  CT M[D + 1][D], t[D + 1][D];
#pragma unroll
  for (int r = 0; r < D; ++r) {
    CT S = F[0][r];
#pragma unroll
    for (int m = 1; m <= D; ++m) S += F[m][r];
#pragma unroll
    for (int m = 0; m <= D; ++m) {
      M[m][r] = S + F[m][r];
      t[m][r] = D == 3 ? fma(CT(4), F[m][r], -S) : CT(4) * F[m][r];
    }
  }
  p2_test<D, CT>(M, t, g, y);
}

// y_K = A_K x_K of one cell, every component.
template <int D, int P, int FORM, bool KP1, typename CT>
__device__ __forceinline__ void cell_action(const PatchArgs& q, const double (&xv)[D + 1][D],
                                            const double (&kap)[D + 1],
                                            const CT (&xc)[FORM == FORM_ELAS ? D : 1][El<D, P>::K],
                                            double (&y)[FORM == FORM_ELAS ? D : 1][El<D, P>::K]) {
  constexpr int NB = D + 1, K = El<D, P>::K, BS = FORM == FORM_ELAS ? D : 1;
  double g[NB][D];
  const double vol = bary_gradients<D>(xv, g);
  if constexpr (P == 2 && sizeof(CT) == 8) {
    if constexpr (FORM == FORM_DIFF) {
      double U[NB][D];
      p2_vertex_gradients<D, double>(xc[0], g, U);
      const double w = vol * q.kscale * (KP1 ? moment3<D>() : moment2<D>());
      if constexpr (KP1) {
        double M[NB][D], t[NB][D];
        double sk = kap[0];
#pragma unroll
        for (int m = 1; m <= D; ++m) sk += kap[m];
#pragma unroll
        for (int r = 0; r < D; ++r) {
          double SU = U[0][r];
#pragma unroll
          for (int m = 1; m <= D; ++m) SU += U[m][r];
          double base = sk * SU;
#pragma unroll
          for (int m = 0; m <= D; ++m) base = fma(kap[m], U[m][r], base);
          double M0 = 0.0;
#pragma unroll
          for (int m = 0; m <= D; ++m) {
            M[m][r] = w * fma(sk, U[m][r], fma(kap[m], fma(2.0, U[m][r], SU), base));
            M0 += M[m][r];
          }
#pragma unroll
          for (int m = 0; m <= D; ++m) t[m][r] = fma(4.0, M[m][r], -M0);
        }
        p2_test<D, double>(M, t, g, y[0]);
      } else {
#pragma unroll
        for (int m = 0; m <= D; ++m)
#pragma unroll
          for (int r = 0; r < D; ++r) U[m][r] *= w;
        p2_test_linear<D, double>(U, g, y[0]);
      }
    } else {
      // stress at the vertices: lambda div(u) I + mu (grad u + grad u^T)
      double sg[NB][D][D];
#pragma unroll
      for (int e = 0; e < D; ++e) {
        double U[NB][D];
        p2_vertex_gradients<D, double>(xc[e], g, U);
#pragma unroll
        for (int m = 0; m <= D; ++m)
#pragma unroll
          for (int d = 0; d < D; ++d) sg[m][e][d] = U[m][d];
      }
      const double w = vol * moment2<D>();
#pragma unroll
      for (int m = 0; m <= D; ++m) {
        double div = sg[m][0][0];
#pragma unroll
        for (int d = 1; d < D; ++d) div += sg[m][d][d];
        const double l = w * q.lmbda * div, mu = w * q.mu;
#pragma unroll
        for (int c = 0; c < D; ++c)
#pragma unroll
          for (int d = c; d < D; ++d) {
            const double s = mu * (sg[m][c][d] + sg[m][d][c]) + (c == d ? l : 0.0);
            sg[m][c][d] = sg[m][d][c] = s;
          }
      }
#pragma unroll
      for (int c = 0; c < D; ++c) {
        double F[NB][D];
#pragma unroll
        for (int m = 0; m <= D; ++m)
#pragma unroll
          for (int d = 0; d < D; ++d) F[m][d] = sg[m][c][d];
        p2_test_linear<D, double>(F, g, y[c]);
      }
    }
  } else if constexpr (P == 2 && FORM == FORM_DIFF && !KP1) {
    // A linear flux, in FP32 up to the factor |T| kappa.  Measured on B200 against
    // the five-point rule (ms per action): P2 tets n=64 0.070 against 0.086, P2
    // triangles n=700 0.031 against 0.037; error 5.3e-8 against 8.2e-8 (rms,
    // random x) and 2.6e-7 against 3.5e-7 (smooth x).
    CT gc[NB][D], U[NB][D], yc[K];
#pragma unroll
    for (int a = 0; a < NB; ++a)
#pragma unroll
      for (int r = 0; r < D; ++r) gc[a][r] = CT(g[a][r]);
    p2_vertex_gradients<D, CT>(xc[0], gc, U);
    p2_test_linear<D, CT>(U, gc, yc);
    const double w = vol * q.kscale * moment2<D>();
#pragma unroll
    for (int j = 0; j < K; ++j) y[0][j] = w * double(yc[j]);
  } else {
    // quadrature (P1: the centroid), in the contraction type
    using Q = Quad<D, P == 1 ? 1 : (FORM == FORM_ELAS ? 2 : 3)>;
    CT gc[NB][D];
#pragma unroll
    for (int a = 0; a < NB; ++a)
#pragma unroll
      for (int r = 0; r < D; ++r) gc[a][r] = CT(g[a][r]);
#pragma unroll
    for (int e = 0; e < BS; ++e)
#pragma unroll
      for (int j = 0; j < K; ++j) y[e][j] = 0.0;
#pragma unroll
    for (int n = 0; n < Q::NQ; ++n) {
      double l[NB];
#pragma unroll
      for (int a = 0; a < NB; ++a) l[a] = Q::lam(n, a);
      const double wq = Q::w(n) * vol;
      CT gu[BS][D];
#pragma unroll
      for (int e = 0; e < BS; ++e) {
#pragma unroll
        for (int d = 0; d < D; ++d) gu[e][d] = CT(0);
#pragma unroll
        for (int a = 0; a < NB; ++a) {
          const CT u = node_derivative<D, P, CT>(xc[e], l, a);
#pragma unroll
          for (int d = 0; d < D; ++d) gu[e][d] = fma(u, gc[a][d], gu[e][d]);
        }
      }
#pragma unroll
      for (int c = 0; c < BS; ++c) {
        CT flux[D];
        if constexpr (FORM == FORM_ELAS) {
          CT div = gu[0][0];
#pragma unroll
          for (int d = 1; d < D; ++d) div += gu[d][d];
#pragma unroll
          for (int d = 0; d < D; ++d) flux[d] = CT(q.mu) * (gu[c][d] + gu[d][c]);
          flux[c] = fma(CT(q.lmbda), div, flux[c]);
        } else {
          double k = q.kscale;
          if constexpr (KP1) {
            double kq = 0.0;
#pragma unroll
            for (int a = 0; a < NB; ++a) kq = fma(kap[a], l[a], kq);
            k *= kq;
          }
#pragma unroll
          for (int d = 0; d < D; ++d) flux[d] = CT(k) * gu[0][d];
        }
        CT S[NB];
#pragma unroll
        for (int a = 0; a < NB; ++a) {
          CT sa = flux[0] * gc[a][0];
#pragma unroll
          for (int d = 1; d < D; ++d) sa = fma(flux[d], gc[a][d], sa);
          S[a] = CT(wq) * sa;
        }
        test_basis<D, P, CT>(S, l, y[c]);
      }
    }
  }
}

// Block size and CTAs per SM.  The kernel is bound by latency -- the plan's and
// x's loads at a CTA's start, then dependent shared-memory reads and FP64
// chains -- so small blocks, many of them resident, win.  P2 tets n=96, ms per
// action: 128 threads, five CTAs (96 registers) 0.246; four 0.280; six (80
// registers, spills) 0.295; 96 threads 0.346; 192 threads 0.32-0.35; 256
// threads 0.53.  Elasticity takes 126 registers and four CTAs: 0.089 against
// 0.13 (five) and 0.18 (six).
constexpr int kPatchThreads = 128;
template <int FORM>
constexpr int patch_ctas() {
  return FORM == FORM_ELAS ? 4 : 5;
}
// Doubles of a staged vertex: its coordinates and kappa, for 16-byte reads (P1
// triangles n=1000 with a constant coefficient: 0.0328 ms against 0.0349 with
// four doubles).
template <int D, bool KP1>
constexpr int patch_vertex() {
  return D == 2 && !KP1 ? 2 : 4;
}
template <int D, int P, int FORM, bool KP1, typename CT>
__global__ void __launch_bounds__(kPatchThreads, patch_ctas<FORM>()) k_patch_apply(const PatchArgs q) {
  constexpr int NB = D + 1, K = El<D, P>::K, BS = FORM == FORM_ELAS ? D : 1;
  constexpr int T = kPatchThreads, VS = patch_vertex<D, KP1>();
  extern __shared__ __align__(16) unsigned char smem[];
  // vertex records (x, y, z, kappa), the nodes' x by component (in the
  // contraction type: one conversion a node, not one a cell and node), the
  // staged actions by component and local node (and a zero slot each), the jobs
  double* vs = reinterpret_cast<double*>(smem);
  CT* xs = reinterpret_cast<CT*>(vs + VS * q.nv);
  CT* ys = xs + BS * q.nx;
  const int plane = K * q.stride + 1;
  unsigned char* jobs = smem + PatchPlan::pad16(uint32_t(8 * VS * q.nv + BS * (q.nx + plane) * int(sizeof(CT))));
  const PatchHdr h = patch_header(q.hdr, blockIdx.x);
  // the plan data of a patch that starts later goes to L2 meanwhile (P2 tets
  // n=96 0.246 -> 0.230 ms)
  const uint32_t later = blockIdx.x + q.ahead;
  PatchHdr hn{};
  if (later < gridDim.x) hn = patch_header(q.hdr, later);
  patch_jobs_copy(q, h, jobs);
  // the cells' local nodes are loaded one cell ahead
  PatchCell<K> cn{};
  if (int(threadIdx.x) < h.ncells) cn.load(q, h, threadIdx.x);
  for (int i = threadIdx.x; i < h.nnodes; i += T) {
    const uint32_t node = __ldg(q.nodes + h.node0 + i);
#pragma unroll
    for (int e = 0; e < BS; ++e) xs[e * q.nx + i] = CT(__ldg(q.x + int64_t(e) * q.nnodes + node));
    if (i < h.nverts) {
      double2* v = reinterpret_cast<double2*>(vs + VS * i);
      if constexpr (VS == 2) {
        v[0] = __ldg(reinterpret_cast<const double2*>(q.xw + 4 * size_t(node)));
      } else {
        double a, b, c, d;
        ld_rec4(q.xw + 4 * size_t(node), a, b, c, d);
        v[0] = make_double2(a, b);
        v[1] = make_double2(D == 3 ? c : 0.0, KP1 ? __ldg(q.kappa + node) : 0.0);
      }
    }
  }
  if (threadIdx.x < BS) ys[threadIdx.x * plane + K * q.stride] = CT(0);
  patch_jobs_wait();
  __syncthreads();
  if (later < gridDim.x) patch_prefetch<K>(q, hn);
  for (int c = threadIdx.x; c < h.ncells; c += T) {
    double xv[NB][D], kap[NB], y[BS][K];
    CT xc[BS][K];
#pragma unroll
    for (int a = 0; a < NB; ++a) {
      const double2* v = reinterpret_cast<const double2*>(reinterpret_cast<const char*>(vs) + VS * cn.off(a));
      const double2 lo = v[0];
      xv[a][0] = lo.x;
      xv[a][1] = lo.y;
      kap[a] = 0.0;
      if constexpr (VS == 4) {
        const double2 hi = v[1];
        if constexpr (D == 3) xv[a][2] = hi.x;
        kap[a] = hi.y;
      }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const char* xj = reinterpret_cast<const char*>(xs) + (sizeof(CT) == 8 ? cn.off(j) : cn.off(j) / 2u);
#pragma unroll
      for (int e = 0; e < BS; ++e) xc[e][j] = reinterpret_cast<const CT*>(xj)[e * q.nx];
    }
    if (c + T < h.ncells) cn.load(q, h, c + T);
    cell_action<D, P, FORM, KP1, CT>(q, xv, kap, xc, y);
#pragma unroll
    for (int e = 0; e < BS; ++e)
#pragma unroll
      for (int j = 0; j < K; ++j) ys[e * plane + j * q.stride + c] = CT(y[e][j]);
  }
  __syncthreads();
  const PatchJobs J = patch_jobs(h, jobs);
  const int lane = threadIdx.x & 31;
  for (int g = threadIdx.x >> 5; g < h.ngroups; g += T / 32) {
    const PatchGroup gr = J.groups[g];
    const uint16_t* code = J.codes + gr.code0 + lane;
    double acc[BS];
#pragma unroll
    for (int e = 0; e < BS; ++e) acc[e] = 0.0;
#pragma unroll 4
    for (int t = 0; t < gr.width; ++t) {
      const uint32_t w = sizeof(CT) == 8 ? code[32 * t] : code[32 * t] / 2u;
      const CT* v = reinterpret_cast<const CT*>(reinterpret_cast<const char*>(ys) + w);
#pragma unroll
      for (int e = 0; e < BS; ++e) acc[e] += double(v[e * plane]);
    }
    if (lane < gr.live) {
      const uint32_t d = J.dest[32 * g + lane];
      double* out = d & kPatchPartial ? q.partial + (d & ~kPatchPartial) : q.y + d;
      const int64_t step = d & kPatchPartial ? q.npartial : q.nnodes;
#pragma unroll
      for (int e = 0; e < BS; ++e) out[e * step] = acc[e];
    }
  }
}

template <int D, int P, int FORM, bool KP1, typename CT>
void run_patch_apply(const PatchPlan& B, const PatchArgs& q, cudaStream_t s) {
  constexpr int K = El<D, P>::K, BS = FORM == FORM_ELAS ? D : 1;
  if (B.npatches > 0) {
    auto kern = k_patch_apply<D, P, FORM, KP1, CT>;
    static unsigned long long configured = 0;
    allow_dynamic_smem(kern, configured);
    const size_t smem = PatchPlan::pad16(uint32_t(8 * patch_vertex<D, KP1>() * q.nv + BS * (q.nx + K * q.stride + 1) * int(sizeof(CT)))) +
                        size_t(B.max_chunks) * 16;
    kern<<<unsigned(B.npatches), kPatchThreads, smem, s>>>(q);
    count_launch();
    check_cuda("patch apply launch");
  }
  if (B.nshared > 0) {
    k_patch_sum<BS><<<unsigned((B.nshared + 255) / 256), 256, 0, s>>>(B.d_shared.as<uint32_t>(), B.d_shared_ptr.as<uint32_t>(),
                                                                      B.nshared, q.partial, B.npartial, q.y, q.nnodes);
    count_launch();
    check_cuda("patch sum launch");
  }
}

}  // namespace dev

dev::PatchView patch_view(const PatchPlan& B, int ctas) {
  dev::PatchView q{};
  q.hdr = B.d_hdr.as<PatchHdr>();
  q.conn = B.d_conn.as<uint16_t>();
  q.nodes = B.d_nodes.as<uint32_t>();
  q.chunks = B.d_chunks.as<uint4>();
  q.npartial = B.npartial;
  q.stride = B.stride;
  q.nx = (B.max_nodes + 1) & ~1;  // (what lies behind starts on 16 bytes)
  q.nv = B.max_verts;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  q.ahead = uint32_t(sms * ctas);
  return q;
}

void launch_patch_apply(const Pattern& P, const dev::AsmParams& p, bool elas, bool kp1, bool fp32, const double* x,
                        double* y, void* stream) {
  const PatchPlan& B = patch_plan(P);
  dev::PatchArgs q{};
  static_cast<dev::PatchView&>(q) = patch_view(B, elas ? dev::patch_ctas<dev::FORM_ELAS>() : dev::patch_ctas<dev::FORM_DIFF>());
  q.xw = p.xw;
  q.kscale = p.kscale;
  q.mu = p.mu;
  q.lmbda = p.lmbda;
  const int64_t n = P.V->dim();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CallScratch work(P, stream);
  q.partial = work.take(&PatchPlan::Work::partial, B.npartial * P.bs);
  // a patch writes its finished nodes while others still read x and kappa, and
  // reads them through the read-only path: one that shares memory with y is
  // copied first
  auto apart = [&](const double* v, int64_t m, DeviceBuffer PatchPlan::Work::*kept) {
    if (!overlap(y, n, v, m)) return v;
    double* c = work.take(kept, m);
    cudaMemcpyAsync(c, v, size_t(m) * sizeof(double), cudaMemcpyDeviceToDevice, s);
    check_cuda("copy of an input of the action");
    return static_cast<const double*>(c);
  };
  x = apart(x, n, &PatchPlan::Work::x);
  if (kp1) q.kappa = apart(p.kappa, P.V->mesh->nv, &PatchPlan::Work::kappa);
  q.x = x;
  q.y = y;
  q.nnodes = p.nnodes;
  const int D = P.V->mesh->tdim, deg = P.V->degree;
  if (elas) {
    if (deg == 1) {
      if (fp32) dev::run_patch_apply<3, 1, dev::FORM_ELAS, false, float>(B, q, s);
      else dev::run_patch_apply<3, 1, dev::FORM_ELAS, false, double>(B, q, s);
    } else {
      if (fp32) dev::run_patch_apply<3, 2, dev::FORM_ELAS, false, float>(B, q, s);
      else dev::run_patch_apply<3, 2, dev::FORM_ELAS, false, double>(B, q, s);
    }
    return;
  }
#define DB2_PA(D_, P_)                                                                   \
  if (D == D_ && deg == P_) {                                                            \
    if (kp1) {                                                                           \
      if (fp32) dev::run_patch_apply<D_, P_, dev::FORM_DIFF, true, float>(B, q, s);      \
      else dev::run_patch_apply<D_, P_, dev::FORM_DIFF, true, double>(B, q, s);          \
    } else {                                                                             \
      if (fp32) dev::run_patch_apply<D_, P_, dev::FORM_DIFF, false, float>(B, q, s);     \
      else dev::run_patch_apply<D_, P_, dev::FORM_DIFF, false, double>(B, q, s);         \
    }                                                                                    \
    return;                                                                              \
  }
  DB2_PA(3, 1) DB2_PA(3, 2) DB2_PA(2, 1) DB2_PA(2, 2)
#undef DB2_PA
}

}  // namespace db2
