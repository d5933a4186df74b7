// patch_load.cu -- the load vector b_i = int f phi_i (f constant or P1) over cell
// patches: a thread per cell computes its volume and loads once into shared
// memory, where the patch's nodes sum them in ascending cell order; nodes shared
// between patches add their partial sums in patch order.  A thread per row
// (k_assemble_vector, which small meshes keep: one launch instead of two)
// rebuilds every incident cell's geometry -- ten times a cell for P2 tetrahedra.
#include <cuda_runtime.h>

#include <optional>
#include <utility>

#include "patch.cuh"

namespace db2 {
namespace dev {

struct PatchLoadArgs : PatchView {
  int bs;
  // of a row range (RANGED): the patches that may hold its rows, the rows, their
  // partial slots, and which kinds of nodes are among them
  const uint32_t* list;
  uint32_t row_begin, row_end, slot_begin, slot_end;
  bool verts, edges;
};

template <int D, int P, int LOADM, int LI>
__device__ __forceinline__ void stage_load(const AsmParams& p, double vol, const double (&fv)[D + 1], double* ys,
                                           int stride) {
  constexpr uint32_t code = perm_code(D, LI);
  double fc[D + 1], unused[D + 1];
#pragma unroll
  for (int a = 0; a <= D; ++a) fc[a] = fv[(code >> (2 * a)) & 3u];
  Geometry<D> G;
  G.vol = vol;
  // (a constant's components are applied to the sums)
  using R = Rows<D, P, double>;
  if constexpr (LOADM == LOAD_CONST) {
    if constexpr (P == 2 && (LI > D)) ys[LI * stride] = vol * R::e_f1();
    else ys[LI * stride] = vol * R::v_f1();
  } else {
    ys[LI * stride] = load_row<D, P, LOADM>(p, G, LI <= D, 0, fc, unused);
  }
}
template <int D, int P, int LOADM, bool RANGED, int... LI>
__device__ __forceinline__ void stage_loads(const AsmParams& p, const PatchLoadArgs& q, double vol,
                                            const double (&fv)[D + 1], double* ys, std::integer_sequence<int, LI...>) {
  auto wanted = [&](bool vertex) { return !RANGED || (vertex ? q.verts : q.edges); };
  ((wanted(LI <= D) ? stage_load<D, P, LOADM, LI>(p, vol, fv, ys, q.stride) : void()), ...);
}

__device__ __forceinline__ void put_load(const AsmParams& p, int c, int64_t node, double v) {
  double* bp = p.b + (int64_t(c) * p.bstride + node - p.bbase);
  *bp = p.add_values ? *bp + v : v;
}

constexpr int kLoadThreads = 128;
// RANGED, the rows of a row range alone: what no row of it takes is neither
// staged nor summed.
template <int D, int P, int LOADM, bool RANGED>
__global__ void __launch_bounds__(kLoadThreads, 5) k_patch_load(const AsmParams p, const PatchLoadArgs q) {
  constexpr int NB = D + 1, K = El<D, P>::K, T = kLoadThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  // vertex records (x, y, z, f), the staged loads by local node (and a zero
  // slot), the jobs
  double* vs = reinterpret_cast<double*>(smem);
  double* ys = vs + 4 * q.nv;
  unsigned char* jobs = smem + PatchPlan::pad16(uint32_t((4 * q.nv + K * q.stride + 1) * 8));
  auto patch = [&](uint32_t i) { return RANGED ? __ldg(q.list + i) : i; };
  const PatchHdr h = patch_header(q.hdr, patch(blockIdx.x));
  const uint32_t later = blockIdx.x + q.ahead;
  PatchHdr hn{};
  if (later < gridDim.x) hn = patch_header(q.hdr, patch(later));
  patch_jobs_copy(q, h, jobs);
  PatchCell<K> cn{};
  if (int(threadIdx.x) < h.ncells) cn.load(q, h, threadIdx.x);
  for (int i = threadIdx.x; i < h.nverts; i += T) {
    const uint32_t node = __ldg(q.nodes + h.node0 + i);
    double a, b, c, d;
    ld_rec4(p.xw + 4 * size_t(node), a, b, c, d);
    double2* v = reinterpret_cast<double2*>(vs + 4 * i);
    v[0] = make_double2(a, b);
    v[1] = make_double2(D == 3 ? c : 0.0, LOADM == LOAD_P1 ? __ldg(p.f + node) : 0.0);
  }
  if (threadIdx.x == 0) ys[K * q.stride] = 0.0;
  patch_jobs_wait();
  __syncthreads();
  if (later < gridDim.x) patch_prefetch<K>(q, hn);
  for (int c = threadIdx.x; c < h.ncells; c += T) {
    double x[NB][D], fv[NB];
#pragma unroll
    for (int a = 0; a < NB; ++a) {
      const double2* v = reinterpret_cast<const double2*>(reinterpret_cast<const char*>(vs) + 4 * cn.off(a));
      const double2 lo = v[0], hi = v[1];
      x[a][0] = lo.x;
      x[a][1] = lo.y;
      if constexpr (D == 3) x[a][2] = hi.x;
      fv[a] = hi.y;
    }
    if (c + T < h.ncells) cn.load(q, h, c + T);
    Geometry<D> G;
    geometry(x, G);
    stage_loads<D, P, LOADM, RANGED>(p, q, G.vol, fv, ys + c, std::make_integer_sequence<int, K>{});
  }
  __syncthreads();
  const PatchJobs J = patch_jobs(h, jobs);
  const int lane = threadIdx.x & 31;
  for (int g = threadIdx.x >> 5; g < h.ngroups; g += T / 32) {
    const PatchGroup gr = J.groups[g];
    uint32_t d = 0;
    bool mine = lane < gr.live;
    if (RANGED) {
      if (mine) {
        d = J.dest[32 * g + lane];
        const uint32_t t = d & ~kPatchPartial;
        mine = d & kPatchPartial ? t >= q.slot_begin && t < q.slot_end : t >= q.row_begin && t < q.row_end;
      }
      if (!__any_sync(0xffffffffu, mine)) continue;
    }
    const uint16_t* code = J.codes + gr.code0 + lane;
    double s = 0.0;
#pragma unroll 4
    for (int t = 0; t < gr.width; ++t)
      s += *reinterpret_cast<const double*>(reinterpret_cast<const char*>(ys) + code[32 * t]);
    if (mine) {
      if (!RANGED) d = J.dest[32 * g + lane];
      if (d & kPatchPartial) {
        q.partial[d & ~kPatchPartial] = s;
      } else {
        for (int c = 0; c < q.bs; ++c) put_load(p, c, d, LOADM == LOAD_CONST ? s * p.fc[c] : s);
      }
    }
  }
}

template <int LOADM>
__global__ void __launch_bounds__(256) k_patch_load_sum(const AsmParams p, const PatchLoadArgs q,
                                                        const uint32_t* __restrict__ shared,
                                                        const uint32_t* __restrict__ ptr, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t node = __ldg(shared + i);
  double s = 0.0;
  const uint32_t s1 = __ldg(ptr + i + 1);
  for (uint32_t t = __ldg(ptr + i); t < s1; ++t) s += __ldg(q.partial + t);
  for (int c = 0; c < q.bs; ++c) put_load(p, c, node, LOADM == LOAD_CONST ? s * p.fc[c] : s);
}

template <int D, int P, int LOADM, bool RANGED>
void launch_patches(const PatchPlan& B, int64_t npatches, const AsmParams& p, const PatchLoadArgs& q, cudaStream_t s) {
  constexpr int K = El<D, P>::K;
  auto kern = k_patch_load<D, P, LOADM, RANGED>;
  static unsigned long long configured = 0;
  allow_dynamic_smem(kern, configured);
  const size_t smem =
      PatchPlan::pad16(uint32_t((4 * q.nv + K * q.stride + 1) * 8)) + size_t(B.max_chunks) * 16;
  if (npatches > 0) {
    kern<<<unsigned(npatches), kLoadThreads, smem, s>>>(p, q);
    count_launch();
    check_cuda("patch load launch");
  }
}

template <int D, int P, int LOADM>
void run_patch_load(const PatchPlan& B, const PatchPlan::RowSet* rows, const AsmParams& p, const PatchLoadArgs& q,
                    cudaStream_t s) {
  if (rows) launch_patches<D, P, LOADM, true>(B, rows->npatches, p, q, s);
  else launch_patches<D, P, LOADM, false>(B, B.npatches, p, q, s);
  const uint32_t s0 = rows ? rows->shared0 : 0;
  const int64_t n = rows ? rows->shared1 - s0 : B.nshared;
  if (n > 0) {
    k_patch_load_sum<LOADM><<<unsigned((n + 255) / 256), 256, 0, s>>>(p, q, B.d_shared.as<uint32_t>() + s0,
                                                                      B.d_shared_ptr.as<uint32_t>() + s0, n);
    count_launch();
    check_cuda("patch load sum launch");
  }
}

}  // namespace dev

bool launch_patch_load(const Pattern& P, const dev::AsmParams& p, int loadm, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // A graph's replays may overlap one another and later calls, so a captured
  // call would need partial sums of its own for the graph's life.
  if (stream_is_capturing(stream)) return false;
  const PatchPlan* plan = patch_plan_for_loads(P);
  if (!plan) return false;
  const PatchPlan& B = *plan;
  std::optional<CallScratch> work;
  double* partial = nullptr;
  std::shared_ptr<const PatchPlan::RowSet> rows;
  try {
    rows = row_set(P);
    work.emplace(P, stream);
    partial = work->take(&PatchPlan::Work::partial, B.npartial);
  } catch (const Error& e) {
    if (e.code != DB2_ERR_NOMEM) throw;
    return false;  // no room for the partial sums: this call by rows
  }
  const int D = P.V->mesh->tdim, deg = P.V->degree;
  dev::PatchLoadArgs q{};
  static_cast<dev::PatchView&>(q) = patch_view(B, 5);
  q.partial = partial;
  q.bs = P.bs;
  if (rows) {
    q.list = rows->list.as<uint32_t>();
    q.row_begin = uint32_t(rows->begin);
    q.row_end = uint32_t(rows->end);
    q.slot_begin = rows->slot0;
    q.slot_end = rows->slot1;
    q.verts = rows->verts;
    q.edges = rows->edges;
  }
#define DB2_PL(D_, P_)                                                                           \
  if (D == D_ && deg == P_) {                                                                    \
    if (loadm == dev::LOAD_CONST) dev::run_patch_load<D_, P_, dev::LOAD_CONST>(B, rows.get(), p, q, s); \
    else dev::run_patch_load<D_, P_, dev::LOAD_P1>(B, rows.get(), p, q, s);                     \
    return true;                                                                                 \
  }
  DB2_PL(3, 1) DB2_PL(3, 2) DB2_PL(2, 1) DB2_PL(2, 2)
#undef DB2_PL
  return false;
}

}  // namespace db2
