// kernels.cu -- launchers of the assembly, vector, action and adjoint kernels.
#include <cuda_runtime.h>

#include "launch.cuh"

namespace db2 {
bool launch_patch_load(const Pattern& P, const dev::AsmParams& p, int loadm, void* stream);  // false: not taken

namespace dev {

// Vector-only assembly (Assembler::assemble for a rank-1 form): one thread
// per dof (component c, node i) gathering its incident cells in cell order.
template <int D, int P, int LOADM>
__global__ void __launch_bounds__(256) k_assemble_vector(const AsmParams p, int bs, int64_t n0,
                                                         int64_t nrange) {
  const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= nrange * bs) return;
  const int c = int(r / nrange);
  const int64_t node = n0 + (r - int64_t(c) * nrange);
  double bsum = 0.0;
  const uint32_t i0 = __ldg(p.inc_ptr + node);
  const uint32_t cnt = __ldg(p.inc_ptr + node + 1) - i0;
  const uint32_t rbase = __ldg(p.rec_goff + (node >> 5)) + uint32_t(node & 31);
  const RowFix<D> F = load_row_fix<D, P, LOADM == LOAD_P1>(p, uint32_t(node));
  for (uint32_t m = 0; m < cnt; ++m) {
    const Rec<D, P> r = load_rec<D, P>(p, rbase + 32u * m);
    double x[D + 1][D], kap[D + 1], fv[D + 1];
    record_cell<D, P, LOADM == LOAD_P1>(p, F, r, i0 + m, x, kap, fv);
    Geometry<D> G;
    geometry(x, G);
    bsum += load_row<D, P, LOADM>(p, G, F.nfix == 1, c, fv, kap);
  }
  double* bp = p.b + int64_t(c) * p.bstride + node - p.bbase;
  *bp = p.add_values ? *bp + bsum : bsum;
}

// Vertex records for one call: the w slots of (x, y, z, w) carry kappa (3D);
// 2D records are (x, y, kappa, f).
__global__ void k_pack_vertex_records(double* __restrict__ xw, int64_t nv, int tdim,
                                      const double* __restrict__ kappa,
                                      const double* __restrict__ f) {
  const int64_t v = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  if (tdim == 3) {
    xw[4 * v + 3] = kappa ? kappa[v] : 0.0;
  } else {
    xw[4 * v + 2] = kappa ? kappa[v] : 0.0;
    xw[4 * v + 3] = f ? f[v] : 0.0;
  }
}

}  // namespace dev

// Writes kappa (and f in 2D) into the mesh's vertex records on `stream`.
void pack_vertex_records(const Pattern& P, const double* kappa, const double* f, void* stream) {
  const Mesh& m = *P.V->mesh;
  if (!kappa && !(m.tdim == 2 && f)) return;
  const int threads = 256;
  dev::k_pack_vertex_records<<<unsigned((m.nv + threads - 1) / threads), threads, 0,
                               static_cast<cudaStream_t>(stream)>>>(
      m.d_x.as<double>(), m.nv, m.tdim, kappa, f);
  count_launch();
  check_cuda("pack_vertex_records launch");
}

dev::AsmParams make_params(const Pattern& P) {
  const_cast<Pattern&>(P).ensure_device();
  dev::AsmParams p{};
  const Mesh& m = *P.V->mesh;
  p.tiles = P.d_tiles.as<Tile>();
  p.node_rowptr = P.d_node_rowptr.as<int32_t>();
  p.inc_ptr = P.d_inc_ptr.as<uint32_t>();
  p.rec = P.d_rec.as<unsigned char>();
  p.rec_goff = P.d_rec_goff.as<uint32_t>();
  p.rec_first = P.d_rec_first.as<unsigned char>();
  p.inc = P.d_inc.as<uint32_t>();
  p.cols = P.d_cols.as<int32_t>();
  p.edge_v = P.V->d_edge_vertices.as<uint32_t>();
  p.nverts = m.nv;
  p.cells = m.d_cells.as<uint32_t>();
  p.xw = m.d_x.as<double>();
  p.cell_nodes = P.V->d_cell_nodes.as<uint32_t>();
  p.cell_inc = P.d_cell_inc.as<uint32_t>();
  p.kscale = 1.0;
  p.fc[0] = p.fc[1] = p.fc[2] = 0.0;
  p.nnz_node = P.nnz_node;
  p.nnodes = P.V->nnodes;
  const OutputLayout o = output_layout(P);
  p.vstride = o.vstride;
  p.vbase = o.vbase;
  p.bstride = o.bstride;
  p.bbase = o.bbase;
  return p;
}

// kappa of a bilinear form -> (uses P1 field, scale)
static bool matrix_coeff(const FormArgs& a, dev::AsmParams& p) {
  switch (a.f.coeff) {
    case DB2_COEFF_NONE: p.kscale = 1.0; return false;
    case DB2_COEFF_CONSTANT: p.kscale = a.f.constant[0]; return false;
    case DB2_COEFF_P1:
    case DB2_COEFF_P1_SCALED:
      if (!a.w) fail(DB2_ERR_ARGUMENT, "form coefficient is a P1 Function but no field was given");
      p.kappa = a.w;
      p.kscale = a.f.coeff == DB2_COEFF_P1 ? 1.0 : a.f.constant[0];
      return true;
    default: fail(DB2_ERR_ARGUMENT, "unknown coefficient kind %d", a.f.coeff);
  }
}

static int load_mode(const FormArgs* L, int bs, dev::AsmParams& p) {
  if (!L) return dev::LOAD_NONE;
  if (L->f.kind != DB2_FORM_LOAD) fail(DB2_ERR_ARGUMENT, "linear form must be DB2_FORM_LOAD");
  switch (L->f.coeff) {
    case DB2_COEFF_NONE:
      for (int c = 0; c < 3; ++c) p.fc[c] = 1.0;
      return dev::LOAD_CONST;
    case DB2_COEFF_CONSTANT:
      for (int c = 0; c < 3; ++c) p.fc[c] = bs == 1 ? L->f.constant[0] : L->f.constant[c];
      return dev::LOAD_CONST;
    case DB2_COEFF_P1:
    case DB2_COEFF_P1_SCALED:
      if (bs != 1) fail(DB2_ERR_UNSUPPORTED, "P1 load coefficient on a vector space");
      if (!L->w) fail(DB2_ERR_ARGUMENT, "load coefficient is a P1 Function but no field was given");
      p.f = L->w;
      p.fc[0] = L->f.coeff == DB2_COEFF_P1 ? 1.0 : L->f.constant[0];
      return dev::LOAD_P1;
    case DB2_COEFF_P1_KAPPA:
      if (bs != 1) fail(DB2_ERR_UNSUPPORTED, "kappa-weighted load on a vector space");
      if (!L->w) fail(DB2_ERR_ARGUMENT, "kappa-weighted load: no field f was given");
      p.f = L->w;
      p.fc[0] = L->f.constant[0];
      return dev::LOAD_KP1;
    default: fail(DB2_ERR_ARGUMENT, "unknown coefficient kind %d", L->f.coeff);
  }
}

// Incidences (row, cell, trial and test component) up to which a pattern is
// assembled for latency: VAR_LAT, one launch instead of a packing launch and
// one per tile class with its fork and join.  Below the line the call's time is
// launches and one row walk; above it the row walks' throughput, where the
// extra registers cost residency.  Measured on B200 (us a call, tile classes ->
// one launch): P2 tets n=10 36 -> 14, n=22 (0.64 M incidences) 37 -> 19, n=26
// (1.05 M) 40 -> 36, n=36 (2.8 M) 78 -> 79; P1 tets n=34 (0.94 M) 23 -> 18, n=38
// (1.3 M) 21 -> 21, n=44 (2.0 M) 31 -> 38; vector P2 elasticity n=12 (0.93 M)
// 35 -> 25, n=14 (1.5 M) 35 -> 35; P2 triangles n=200 (0.48 M) 21 -> 14, n=300
// (1.08 M) 29 -> 30.  P2 tets in FP32 (74 to 80 registers in
// the tile classes, no spills) gain longer in a loop, a call after which the host
// waits does not: n=34 (2.4 M) 71 -> 59 and alone 74 -> 73, n=35 (2.6 M) 73 -> 67
// and 76 -> 81, n=36 78 -> 69 and 80 -> 83; elasticity n=16 (2.2 M) 51 -> 48 and
// 62 -> 61, n=18 (3.1 M) 67 -> 66 and 78 -> 77.  By the pattern's size, not the row
// range's, so that a range's rows equal the whole assembly's bit for bit.
static bool latency_bound(const Pattern& P, bool fp32) {
  const int64_t incidences = int64_t(P.inc.size()) * P.bs * P.bs;
  const int64_t line = P.V->mesh->tdim == 2 ? 1000000 : fp32 && P.V->degree == 2 ? 2400000 : 1400000;
  return incidences <= line && P.rec_escapes == 0;
}

// Load vectors over cell patches (patch_load.cu: two launches, every cell once)
// or by the thread-per-row kernel (one launch, in 2D with a P1 f after a packing
// one): the incidences from which the patches are no slower.  A row's work is
// the cells around it, once for each component; its kernel is short where a
// cell's load is one number (constant f) and its geometry cheap (triangles, few
// cells a row in P1).  Measured on B200, us a call in a loop, by rows / over
// patches, on both sides of each line:
//   P1 tets  f P1   n=33 (0.86 M) 14.6 / 15.7, n=34 (0.94 M) 16.5 / 15.8
//            const  n=52 (3.4 M) 20.6 / 23.2, n=56 (4.2 M) 26.7 / 26.7, n=64 49 / 35
//            vector n=28 (0.53 M) 14.4 / 15.4, n=30 (0.65 M) 16.6 / 15.5
//   P2 tets  f P1   n=14 (0.16 M) 17.3 / 15.6, n=24 20.6 / 15.6, n=96 531 / 200
//            const  n=15 (0.20 M) 14.4 / 15.2, n=18 (0.35 M) 16.4 / 15.2, n=96 431 / 201
//            vector n=10 (60,000) 14.8 / 15.3, n=18 (0.35 M) 18.5 / 15.1
//   P1 tris  f P1   n=700 (2.9 M) 22.0 / 22.6, n=750 (3.4 M) 24.7 / 24.6, n=850 31 / 26.7
//            const  n=850 (4.3 M) 20.5 / 26.7, n=1150 (7.9 M) 40 / 58: always by rows
//            vector n=500 (1.5 M) 14.6 / 15.5, n=550 (1.8 M) 16.5 / 16.3, n=650 21.7 / 18.5
//   P2 tris  f P1   n=300 (1.1 M) 16.3 / 15.5, n=360 (1.6 M) 18.5 / 16.0, n=500 30.5 / 18.8
//            const  n=350 (1.5 M) 12.4 / 15.4, n=460 (2.5 M) 18.5 / 18.5, n=500 (3 M) 23.7 / 20.6
//            vector n=300 (1.1 M) 16.5 / 15.2, n=400 (1.9 M) 26.7 / 16.5
// By the pattern's size, not the row range's, so that a range's rows equal the
// whole vector's bit for bit; one eighth of P2 n=96's rows (set_row_range) takes
// 29-43 us against 49-60 by rows, the eighth that holds the vertices, which
// meet every patch, 145 against 150 (constant f) and 178 (P1 f).
static bool load_over_patches(const Pattern& P, int loadm) {
  const int tdim = P.V->mesh->tdim, kind = loadm == dev::LOAD_P1 ? 0 : P.bs == 1 ? 1 : 2;
  static const int64_t kLine[2][2][3] = {{{3400000, INT64_MAX, 1800000}, {1500000, 2700000, 1500000}},
                                         {{900000, 4500000, 640000}, {200000, 300000, 200000}}};
  return int64_t(P.inc.size()) >= kLine[tdim - 2][P.V->degree - 1][kind];
}

// Whether the call writes over the memory of its kappa or f.  The tile classes
// and the row kernel have copied them to the vertex records before they write
// (f on triangles only); what reads the arrays beside its writes must not run.
static bool writes_coefficients(const Pattern& P, const dev::AsmParams& p) {
  int64_t nrows = P.nrows, nnz = P.nnz;
  if (P.block_storage) row_block_size(P, &nrows, &nnz);
  const int64_t nv = P.V->mesh->nv;
  return overlap(p.b, nrows, p.kappa, nv) || overlap(p.b, nrows, p.f, nv) || overlap(p.vals, nnz, p.kappa, nv) ||
         overlap(p.vals, nnz, p.f, nv);
}

void launch_assemble(const Pattern& P, const FormArgs* a, const FormArgs* L, int precision,
                     double* vals, double* b, bool add_values, const uint8_t* bc_flags,
                     const double* bc_vals, void* stream) {
  const Space& V = *P.V;
  const int D = V.mesh->tdim;
  // the tile kernel writes its value segments with 16-byte bulk copies from
  // an 8-byte-aligned base (and doubles elsewhere): refuse other pointers
  // here rather than fault on the device
  if ((reinterpret_cast<uintptr_t>(vals) | reinterpret_cast<uintptr_t>(b)) % alignof(double))
    fail(DB2_ERR_ARGUMENT, "value and vector arrays must be 8-byte aligned device pointers");
  dev::AsmParams p = make_params(P);
  p.vals = vals;
  p.b = b;
  p.add_values = add_values ? 1 : 0;
  p.bc_flags = bc_flags;
  p.bc_vals = bc_vals;
  const int loadm = load_mode(L, P.bs, p);
  if (loadm == dev::LOAD_KP1 && !(a && a->f.kind == DB2_FORM_DIFFUSION &&
                                  (a->f.coeff == DB2_COEFF_P1 || a->f.coeff == DB2_COEFF_P1_SCALED)))
    fail(DB2_ERR_UNSUPPORTED, "a kappa-weighted load (DB2_COEFF_P1_KAPPA) is assembled together with "
         "kappa*grad(u).grad(v)*dx with a P1 kappa (db2_assemble_system / _system_bc)");
  if (!a) {
    // rank-1 form only
    if (loadm == dev::LOAD_NONE) fail(DB2_ERR_ARGUMENT, "nothing to assemble");
    if (load_over_patches(P, loadm) && !writes_coefficients(P, p) && launch_patch_load(P, p, loadm, stream)) return;
    pack_vertex_records(P, nullptr, loadm == dev::LOAD_P1 ? p.f : nullptr, stream);
    // the node rows of the pattern's row range (all of them by default)
    const int64_t n0 = P.row_begin, nr = (P.row_end < 0 ? V.nnodes : P.row_end) - n0;
    const int64_t n = nr * P.bs;
    if (n == 0) return;
    const int threads = 256;
    const unsigned blocks = unsigned((n + threads - 1) / threads);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define DB2_VEC(D_, P_)                                                                       \
  if (D == D_ && V.degree == P_) {                                                            \
    if (loadm == dev::LOAD_CONST) dev::k_assemble_vector<D_, P_, dev::LOAD_CONST><<<blocks, threads, 0, s>>>(p, P.bs, n0, nr); \
    else dev::k_assemble_vector<D_, P_, dev::LOAD_P1><<<blocks, threads, 0, s>>>(p, P.bs, n0, nr);    \
    count_launch();                                                                           \
    check_cuda("assemble_vector launch");                                                     \
    return;                                                                                   \
  }
    DB2_VEC(3, 1) DB2_VEC(3, 2) DB2_VEC(2, 1) DB2_VEC(2, 2)
#undef DB2_VEC
    fail(DB2_ERR_UNSUPPORTED, "vector assembly not provided for this element");
  }
  if (bc_flags && (!bc_vals || !L || !b)) fail(DB2_ERR_ARGUMENT, "Dirichlet data needs values, a linear form and b");
  p.cols = P.d_cols.as<int32_t>();
  dev::LaunchCfg cfg;
  cfg.class_begin = &P.class_begin;
  cfg.class_smem = &P.class_smem;
  cfg.threads = P.tile_threads;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cfg.escapes = P.rec_escapes > 0;
  const bool fp32 = precision == DB2_FP32_CONTRACT;
  cfg.latency = latency_bound(P, fp32);
  if (precision != DB2_FP64 && precision != DB2_FP32_CONTRACT) fail(DB2_ERR_ARGUMENT, "unknown precision %d", precision);
  bool ok = false;
  if (a->f.kind == DB2_FORM_DIFFUSION) {
    if (P.bs != 1) fail(DB2_ERR_UNSUPPORTED, "diffusion form on a vector space");
    const bool kp1 = matrix_coeff(*a, p);
    cfg.latency = cfg.latency && !writes_coefficients(P, p);
    if (!cfg.latency)
      pack_vertex_records(P, kp1 ? p.kappa : nullptr,
                        (loadm == dev::LOAD_P1 || loadm == dev::LOAD_KP1) ? p.f : nullptr, stream);
    ok = D == 3 ? dev::dispatch_tet_diff(V.degree, p, cfg, kp1, loadm, fp32)
                : dev::dispatch_tri_diff(V.degree, p, cfg, kp1, loadm, fp32);
  } else if (a->f.kind == DB2_FORM_ELASTICITY) {
    if (P.bs != D || D != 3) fail(DB2_ERR_UNSUPPORTED, "elasticity needs a 3D vector space");
    p.mu = a->f.mu;
    p.lmbda = a->f.lmbda;
    if (a->f.coeff != DB2_COEFF_NONE) fail(DB2_ERR_UNSUPPORTED, "elasticity takes no coefficient");
    pack_vertex_records(P, nullptr, nullptr, stream);
    ok = dev::dispatch_tet_elas(V.degree, p, cfg, false, loadm, fp32);
  } else {
    fail(DB2_ERR_ARGUMENT, "bilinear form kind %d not provided", a->f.kind);
  }
  if (!ok) fail(DB2_ERR_UNSUPPORTED, "no kernel for this form/coefficient/load combination");
}

}  // namespace db2
