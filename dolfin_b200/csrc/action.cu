// action.cu -- matrix-free action y = A x (dispatch; patch.cu holds its kernels,
// action_tc.cuh the tensor-core one) and the adjoint (VJP) with respect to a P1
// coefficient.
#include <cuda_runtime.h>

#include "launch.cuh"
#include "adjoint.cuh"
#include "action_tc.cuh"

#include <algorithm>

namespace db2 {
namespace dev {

// The ordered gather behind the tensor-core action: y = sum of the element
// actions of the node's incident cells, in ascending cell order -- a fixed
// order, so the result is bitwise repeatable.  The terms lie in incidence
// order, contiguous for each node.
__global__ void __launch_bounds__(256) k_apply_gather(const uint32_t* __restrict__ inc_ptr, int64_t nnodes,
                                                      const float* __restrict__ ycell, double* __restrict__ y) {
  const int64_t node = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (node >= nnodes) return;
  const uint32_t s0 = __ldg(inc_ptr + node), s1 = __ldg(inc_ptr + node + 1);
  double acc = 0.0;
  for (uint32_t s = s0; s < s1; ++s) acc += double(__ldg(ycell + s));
  y[node] = acc;
}

// A cell's incidences are read at once, in wide loads, and kept, and its vertex
// nodes taken from its vertices; P2 triangles without a load (LATE) read both for
// each node where they are used -- measured on B200, us a VJP, at once / late:
// P2 triangles n=700 94.0 / 90.7 (FP32 97.9 / 93.4), with a load 94.8 / 100.7;
// P1 tets n=64 83 / 93 and 87 / 103, P2 tets n=40 77 / 91 and 84 / 103.
template <int D, int P, bool LOADK>
constexpr bool vjp_late() {
  return D == 2 && P == 2 && !LOADK;
}

// gA at the columns of a cell's row by its incidence record, and gb.
template <int D, int P, bool LOADK>
struct RecordRow {
  const AsmParams& p;
  int64_t cell;
  const uint32_t (&v)[D + 1];          // the cell's vertices
  const uint32_t (&inc)[El<D, P>::K];  // and incidences
  const double* gA;
  const double* gb;
  template <int LI>
  __device__ __forceinline__ void get(double (&g)[El<D, P>::K], double& gbi) const {
    constexpr int K = El<D, P>::K;
    constexpr bool LATE = vjp_late<D, P, LOADK>();
    const uint32_t ii = LATE ? __ldg(p.cell_inc + size_t(cell) * K + LI) : inc[LI];
    // vertex nodes are numbered as the vertices (natural numbering)
    uint32_t node;
    if constexpr (LI <= D && !LATE) node = v[LI];
    else node = __ldg(p.cell_nodes + size_t(cell) * K + LI);
    const double* grow = gA + __ldg(p.node_rowptr + node);
    const Rec<D, P> rr = load_rec<D, P>(p, rec_index<D, P>(p, node, ii - __ldg(p.inc_ptr + node)));
#pragma unroll
    for (int j = 0; j < K; ++j) g[j] = __ldg(grow + rr.slot(j));
    if constexpr (LOADK) gbi = __ldg(gb + node);
  }
};

// Adjoint, step 1 (one thread per cell): t[cell][m] = sum_{i,j in cell}
// gA_ij dA^K_ij/dkappa_m + sum_i gb_i db^K_i/dkappa_m for the P1 kappa
// basis functions m of the cell.  The cell's vertices and geometry are
// loaded and computed once; each local node's relabelled geometry tensor is
// a permutation of the cell's.
// Register caps: the P2 node parts (ten of them, inlined) would take up to
// 174 registers uncapped; P1 cells need no more than 64.
template <int P>
constexpr int vjp_maxnreg() {
  return P == 1 ? 64 : 128;
}
template <int D, int P, bool LOADK, typename CT>
__global__ void __maxnreg__((vjp_maxnreg<P>())) k_vjp_cells(const AsmParams p, int64_t ncells,
                                                   const double* __restrict__ gA,
                                                   const double* __restrict__ gb,
                                                   double* __restrict__ t) {
  using E = El<D, P>;
  constexpr int NB = D + 1;
  const int64_t cell = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (cell >= ncells) return;
  uint32_t v[NB];
  load_verts<D>(p, uint32_t(cell), v);
  // the cell's incidences, in the widest loads its row of the array allows
  uint32_t inc[E::K];
  {
    const uint32_t* ci = p.cell_inc + size_t(cell) * E::K;
    if constexpr (vjp_late<D, P, LOADK>()) {
    } else if constexpr (E::K % 4 == 0) {
#pragma unroll
      for (int j = 0; j < E::K; j += 4) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(ci + j));
        inc[j] = w.x; inc[j + 1] = w.y; inc[j + 2] = w.z; inc[j + 3] = w.w;
      }
    } else if constexpr (E::K % 2 == 0) {
#pragma unroll
      for (int j = 0; j < E::K; j += 2) {
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(ci + j));
        inc[j] = w.x; inc[j + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < E::K; ++j) inc[j] = __ldg(ci + j);
    }
  }
  double x[NB][D], kap_unused[NB], f_unused[NB];
  load_vertex_data<D, false>(p, v, x, kap_unused, f_unused);
  double fv[NB];
#pragma unroll
  for (int a = 0; a < NB; ++a) fv[a] = LOADK ? __ldg(p.f + v[a]) : 0.0;
  Geometry<D> G;
  geometry(x, G);
  double Wn[NB][NB];
#pragma unroll
  for (int a = 0; a < NB; ++a)
#pragma unroll
    for (int b = a; b < NB; ++b) Wn[a][b] = Wn[b][a] = ndot<D>(G, a, b);
  double acc[NB];
#pragma unroll
  for (int a = 0; a < NB; ++a) acc[a] = 0.0;
  const RecordRow<D, P, LOADK> row{p, cell, v, inc, gA, gb};
  vjp_nodes<D, P, LOADK, CT>(p, Wn, G.s, G.vol, fv, row, acc, std::make_integer_sequence<int, E::K>{});
  // in vertex-incidence order (vertex nodes come first in the node-contiguous
  // incidence array), so that step 2 reads each vertex's terms contiguously
#pragma unroll
  for (int a = 0; a < NB; ++a)
    t[vjp_late<D, P, LOADK>() ? __ldg(p.cell_inc + size_t(cell) * E::K + a) : inc[a]] = acc[a];
}

// Adjoint, step 2 (one thread per vertex): dkappa[v] = sum over cells around
// v, in cell order, of their terms for v (contiguous: incidence order).
template <int D, int P>
__global__ void __launch_bounds__(256) k_vjp_vertices(const AsmParams p, int64_t nv,
                                                      const double* __restrict__ t,
                                                      double* __restrict__ dk) {
  const int64_t v = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  double s = 0.0;
  const uint32_t s1 = __ldg(p.inc_ptr + v + 1);
  for (uint32_t ii = __ldg(p.inc_ptr + v); ii < s1; ++ii) s += __ldg(t + ii);
  dk[v] = s;
}

// The FP32-contraction action of P2 diffusion on tetrahedra: element actions
// by the tensor-core kernel (action_tc.cuh), then the same ordered gather.
template <bool KP1>
void run_apply_tc(const Pattern& Pt, const AsmParams& p, const double* x, double* y, cudaStream_t s) {
  const int64_t nc = Pt.V->mesh->nc;
  const size_t need = size_t(nc) * 10 * sizeof(float);
  if (Pt.d_cellvals.bytes < need) Pt.d_cellvals.alloc(need);
  float* ycell = Pt.d_cellvals.as<float>();
  if (nc > 0) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // persistent: the 5 CTAs per SM the launch bounds provide for (registers
    // <= 102; 5 x 30 KB of shared memory; 5 x 64 of the 512 tensor-memory
    // columns)
    const int64_t ntiles = (nc + kTcM - 1) / kTcM;
    const unsigned grid = unsigned(std::min<int64_t>(ntiles, int64_t(sms) * 5));
    k_apply_tc_p2<KP1><<<grid, kTcM, sizeof(TcSmem), s>>>(p, nc, x, ycell);
    count_launch();
    check_cuda("tensor-core apply launch");
  }
  k_apply_gather<<<unsigned((p.nnodes + 255) / 256), 256, 0, s>>>(p.inc_ptr, p.nnodes, ycell, y);
  count_launch();
  check_cuda("apply gather launch");
}

}  // namespace dev

int tensor_core_status() {
  int v = 0;
  const cudaError_t e = cudaMemcpyFromSymbol(&v, dev::g_tc_status, sizeof(int));
  if (e != cudaSuccess) fail(DB2_ERR_CUDA, "reading the tensor-core status: %s", cudaGetErrorString(e));
  return v;
}

dev::AsmParams make_params(const Pattern& P);
void launch_patch_apply(const Pattern& P, const dev::AsmParams& p, bool elas, bool kp1, bool fp32, const double* x,
                        double* y, void* stream);
void pack_vertex_records(const Pattern& P, const double* kappa, const double* f, void* stream);

void launch_apply(const Pattern& P, const FormArgs& a, int precision, const double* x, double* y,
                  void* stream) {
  dev::AsmParams p = make_params(P);
  const int D = P.V->mesh->tdim, deg = P.V->degree;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool tc = precision == DB2_FP32_TENSOR_CORE;
  const bool fp32 = precision == DB2_FP32_CONTRACT || tc;
  if (precision != DB2_FP64 && !fp32) fail(DB2_ERR_ARGUMENT, "unknown precision %d", precision);
  bool kp1 = false;
  if (a.f.kind == DB2_FORM_DIFFUSION) {
    if (P.bs != 1) fail(DB2_ERR_UNSUPPORTED, "diffusion form on a vector space");
    p.kscale = a.f.coeff == DB2_COEFF_CONSTANT || a.f.coeff == DB2_COEFF_P1_SCALED ? a.f.constant[0] : 1.0;
    kp1 = a.f.coeff == DB2_COEFF_P1 || a.f.coeff == DB2_COEFF_P1_SCALED;
    if (kp1 && !a.w) fail(DB2_ERR_ARGUMENT, "P1 coefficient field missing");
    p.kappa = a.w;
    if (!tc) {
      launch_patch_apply(P, p, false, kp1, fp32, x, y, stream);
      return;
    }
    if (D != 3 || deg != 2) fail(DB2_ERR_UNSUPPORTED, "the tensor-core action is for P2 tetrahedra");
    // FP32 contraction on the tensor cores
    pack_vertex_records(P, kp1 ? a.w : nullptr, nullptr, stream);
    if (kp1) dev::run_apply_tc<true>(P, p, x, y, s);
    else dev::run_apply_tc<false>(P, p, x, y, s);
    return;
  } else if (a.f.kind == DB2_FORM_ELASTICITY) {
    if (D != 3 || P.bs != 3) fail(DB2_ERR_UNSUPPORTED, "elasticity needs a 3D vector space");
    if (tc) fail(DB2_ERR_UNSUPPORTED, "the tensor-core action is for P2 diffusion");
    p.mu = a.f.mu;
    p.lmbda = a.f.lmbda;
    launch_patch_apply(P, p, true, false, fp32, x, y, stream);
    return;
  }
  fail(DB2_ERR_UNSUPPORTED, "matrix-free action not provided for this form/element");
}

void preload_vjp_kernels() {
  cudaFuncAttributes at;
  cudaError_t e = cudaSuccess;
  auto get = [&](const void* f) {
    const cudaError_t r = cudaFuncGetAttributes(&at, f);
    if (r != cudaSuccess) e = r;
  };
#define DB2_VJP_LOAD(D_, P_)                                                  \
  get((const void*)dev::k_vjp_cells<D_, P_, true, float>);                    \
  get((const void*)dev::k_vjp_cells<D_, P_, true, double>);                   \
  get((const void*)dev::k_vjp_cells<D_, P_, false, float>);                   \
  get((const void*)dev::k_vjp_cells<D_, P_, false, double>);                  \
  get((const void*)dev::k_vjp_vertices<D_, P_>);
  DB2_VJP_LOAD(3, 1) DB2_VJP_LOAD(3, 2) DB2_VJP_LOAD(2, 1) DB2_VJP_LOAD(2, 2)
#undef DB2_VJP_LOAD
  if (e != cudaSuccess) fail(DB2_ERR_CUDA, "loading the adjoint kernels: %s", cudaGetErrorString(e));
}

size_t vjp_scratch_doubles(const Pattern& P) {
  return size_t(P.V->mesh->nc) * (P.V->mesh->tdim + 1);
}

void launch_vjp(const Pattern& P, const FormArgs& a, const FormArgs& L, int precision,
                const double* gA, const double* gb, double* dkappa, double* scratch,
                void* stream) {
  if (a.f.kind != DB2_FORM_DIFFUSION || P.bs != 1)
    fail(DB2_ERR_UNSUPPORTED, "the adjoint is provided for kappa*grad(u).grad(v)*dx on scalar spaces");
  if (!(a.f.coeff == DB2_COEFF_P1 || a.f.coeff == DB2_COEFF_P1_SCALED))
    fail(DB2_ERR_ARGUMENT, "the adjoint is with respect to a P1 kappa");
  const bool tc = precision == DB2_FP32_TENSOR_CORE;
  const bool fp32 = precision == DB2_FP32_CONTRACT || tc;
  if (precision != DB2_FP64 && !fp32) fail(DB2_ERR_ARGUMENT, "unknown precision %d", precision);
  dev::AsmParams p = make_params(P);
  p.kscale = a.f.coeff == DB2_COEFF_P1_SCALED ? a.f.constant[0] : 1.0;
  p.kappa = a.w;
  // L = kappa * f * v * dx contributes when its coefficient is P1_SCALED
  // (the kappa-weighted load); any other load does not depend on kappa.
  const bool loadk = gb && L.f.kind == DB2_FORM_LOAD &&
                     (L.f.coeff == DB2_COEFF_P1_SCALED || L.f.coeff == DB2_COEFF_P1_KAPPA);
  if (loadk) {
    if (!L.w) fail(DB2_ERR_ARGUMENT, "kappa-weighted load needs its P1 field f");
    p.f = L.w;
    p.fc[0] = L.f.coeff == DB2_COEFF_P1_KAPPA ? L.f.constant[0] : 1.0;
  }
  const int D = P.V->mesh->tdim, deg = P.V->degree;
  const int64_t nc = P.V->mesh->nc, nv = P.V->mesh->nv;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned bc = unsigned((nc + 255) / 256), bv = unsigned((nv + 255) / 256);
#define DB2_VJP(D_, P_)                                                                        \
  if (D == D_ && deg == P_) {                                                                  \
    if (loadk) {                                                                               \
      if (fp32) dev::k_vjp_cells<D_, P_, true, float><<<bc, 256, 0, s>>>(p, nc, gA, gb, scratch); \
      else dev::k_vjp_cells<D_, P_, true, double><<<bc, 256, 0, s>>>(p, nc, gA, gb, scratch);  \
    } else {                                                                                   \
      if (fp32) dev::k_vjp_cells<D_, P_, false, float><<<bc, 256, 0, s>>>(p, nc, gA, gb, scratch); \
      else dev::k_vjp_cells<D_, P_, false, double><<<bc, 256, 0, s>>>(p, nc, gA, gb, scratch); \
    }                                                                                          \
    dev::k_vjp_vertices<D_, P_><<<bv, 256, 0, s>>>(p, nv, scratch, dkappa);                         \
    count_launch(2);                                                                           \
    check_cuda("vjp launch");                                                                  \
    return;                                                                                    \
  }
  DB2_VJP(3, 1) DB2_VJP(3, 2) DB2_VJP(2, 1) DB2_VJP(2, 2)
#undef DB2_VJP
  fail(DB2_ERR_UNSUPPORTED, "adjoint not provided for this element");
}

}  // namespace db2
