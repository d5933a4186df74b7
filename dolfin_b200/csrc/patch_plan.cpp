// patch_plan.cpp -- cell patches of a pattern (PatchPlan, internal.h).
//
// A cell belongs to its first vertex; the vertices are clustered by recursive
// bisection of their coordinates along the longest side, cut at the widest gap
// near the position that fills the patches.  On lattice-like meshes (jittered ones too) the cuts fall
// between lattice planes and patches are boxes, with few nodes shared between
// them; elsewhere they are cut at that position.
#include <cmath>
#include <cstring>
#include <numeric>

#include "internal.h"

namespace db2 {
namespace {

struct Bisector {
  const Mesh& m;
  const std::vector<uint32_t>& cell0;  // first cell (by first vertex) of each vertex
  int max_cells;

  // (zero for a coordinate that is no number or infinite: the order below must be one)
  double coord(int64_t v, int r) const {
    const double x = m.x[v * m.tdim + r];
    return std::isfinite(x) ? x : 0.0;
  }
  int64_t cells_of(const uint32_t* v, int64_t n) const {
    int64_t c = 0;
    for (int64_t i = 0; i < n; ++i) c += cell0[v[i] + 1] - cell0[v[i]];
    return c;
  }
  // Reorders v[0, n), n > 1, and returns the cut (0 < cut < n): as many full
  // patches on one side as on the other, or one more.
  int64_t split(uint32_t* v, int64_t n) const {
    const int D = m.tdim;
    double lo[3], hi[3];
    for (int r = 0; r < D; ++r) lo[r] = hi[r] = coord(v[0], r);
    for (int64_t i = 1; i < n; ++i)
      for (int r = 0; r < D; ++r) {
        const double x = coord(v[i], r);
        lo[r] = std::min(lo[r], x);
        hi[r] = std::max(hi[r], x);
      }
    int axis = 0;
    for (int r = 1; r < D; ++r)
      if (hi[r] - lo[r] > hi[axis] - lo[axis]) axis = r;
    auto key = [&](uint32_t a) { return coord(a, axis); };
    auto less = [&](uint32_t a, uint32_t b) {
      const double p = key(a), q = key(b);
      return p < q || (!(q < p) && a < b);
    };
    const int64_t parts = (cells_of(v, n) + max_cells - 1) / max_cells;
    const int64_t mid = std::min(n - 1, std::max<int64_t>(1, parts > 1 ? n * (parts / 2) / parts : n / 2));
    // the window around it in which the cut may lie
    // (about one lattice plane of n vertices to either side)
    const int64_t w = std::max<int64_t>(1, std::min<int64_t>(n / 6, int64_t(std::pow(double(n), 2.0 / 3.0))));
    const int64_t b = std::max<int64_t>(1, mid - w), e = std::min<int64_t>(n - 1, mid + w);
    if (b >= e) {
      std::nth_element(v, v + mid, v + n, less);
      return mid;
    }
    std::nth_element(v, v + (b - 1), v + n, less);
    std::nth_element(v + b, v + e, v + n, less);
    std::sort(v + b, v + e, less);  // v[b - 1 .. e] now ascending
    int64_t cut = mid;
    double best = -1.0;
    for (int64_t i = b; i <= e; ++i) {
      const double gap = key(v[i]) - key(v[i - 1]);
      const int64_t d = std::abs(i - mid), dc = std::abs(cut - mid);
      if (gap > best * 1.5 || (gap > best / 1.5 && d < dc)) {
        best = std::max(gap, best);
        cut = i;
      }
    }
    return cut;
  }
  void leaves(uint32_t* v, int64_t base, int64_t n, std::vector<int64_t>& ends) const {
    if (n <= 1 || cells_of(v, n) <= max_cells) {
      ends.push_back(base + n);
      return;
    }
    const int64_t c = split(v, n);
    leaves(v, base, c, ends);
    leaves(v + c, base + c, n - c, ends);
  }
};

// Node id -> local number, for one patch at a time (open addressing; clearing
// is a new stamp).
struct NodeTable {
  std::vector<uint32_t> key, stamp, val;
  uint32_t now = 0, mask;
  explicit NodeTable(size_t nodes) {
    size_t n = 64;
    while (n < 2 * nodes) n *= 2;
    key.resize(n);
    stamp.assign(n, 0);
    val.resize(n);
    mask = uint32_t(n - 1);
  }
  void clear() { ++now; }
  size_t find(uint32_t k) const {
    size_t i = (k * 2654435761u >> 7) & mask;
    while (stamp[i] == now && key[i] != k) i = (i + 1) & mask;
    return i;
  }
  bool insert(uint32_t k) {  // true if it was not there
    const size_t i = find(k);
    if (stamp[i] == now) return false;
    stamp[i] = now;
    key[i] = k;
    return true;
  }
};

struct Part {  // patches of a contiguous range of clusters
  std::vector<PatchHdr> hdr;
  std::vector<uint32_t> cells;  // of each patch, ascending
  std::vector<uint32_t> nodes;
  std::vector<uint16_t> conn;
  std::vector<uint8_t> chunks;
  int max_nodes = 0, max_verts = 0, max_chunks = 0;
};

}  // namespace

std::unique_ptr<PatchPlan> make_patches(const Pattern& P, int max_cells) {
  const Space& V = *P.V;
  const Mesh& m = *V.mesh;
  const int k = V.k, nvc = m.tdim + 1, kc = patch_conn(k);
  auto B = std::make_unique<PatchPlan>();
  // 16-bit byte offsets of the staged values and of the local nodes
  max_cells = std::min(max_cells, 8191 / k - 1);
  if (uint64_t(V.nnodes) >= kPatchPartial) fail(DB2_ERR_UNSUPPORTED, "too many nodes for cell patches");
  // cells by first vertex, ascending
  std::vector<uint32_t> cell0(size_t(m.nv) + 1, 0), bucket(static_cast<size_t>(m.nc));
  for (int64_t c = 0; c < m.nc; ++c) cell0[m.cells[c * nvc] + 1]++;
  for (int64_t v = 0; v < m.nv; ++v) cell0[v + 1] += cell0[v];
  {
    std::vector<uint32_t> fill(cell0.begin(), cell0.end() - 1);
    for (int64_t c = 0; c < m.nc; ++c) bucket[fill[m.cells[c * nvc]]++] = uint32_t(c);
  }
  std::vector<uint32_t> vert;
  for (int64_t v = 0; v < m.nv; ++v)
    if (cell0[v + 1] > cell0[v]) vert.push_back(uint32_t(v));
  const Bisector C{m, cell0, max_cells};
  // top levels of the bisection, then the parts in parallel
  std::vector<int64_t> cuts{0, int64_t(vert.size())};
  while (cuts.size() < 256 && m.nc / int64_t(cuts.size()) > 8 * max_cells) {
    std::vector<int64_t> mid(cuts.size() - 1), next{0};
    parallel_for(int64_t(mid.size()), [&](int64_t b, int64_t e) {
      for (int64_t i = b; i < e; ++i) {
        const int64_t n = cuts[i + 1] - cuts[i];
        mid[i] = cuts[i] + (n > 1 ? C.split(vert.data() + cuts[i], n) : 0);
      }
    }, 1);
    for (size_t i = 0; i + 1 < cuts.size(); ++i) {
      if (mid[i] > cuts[i]) next.push_back(mid[i]);
      next.push_back(cuts[i + 1]);
    }
    if (next.size() == cuts.size()) break;
    cuts.swap(next);
  }
  const int64_t nparts = int64_t(cuts.size()) - 1;
  std::vector<Part> parts(static_cast<size_t>(nparts));
  // pass 1: the patches' cells and nodes
  parallel_for(nparts, [&](int64_t b, int64_t e) {
    std::vector<int64_t> ends;
    std::vector<uint32_t> cells;
    NodeTable table(size_t(max_cells) * k);
    for (int64_t i = b; i < e; ++i) {
      Part& T = parts[i];
      ends.clear();
      C.leaves(vert.data() + cuts[i], cuts[i], cuts[i + 1] - cuts[i], ends);
      int64_t at = cuts[i];
      for (int64_t end : ends) {
        cells.clear();
        for (; at < end; ++at)
          cells.insert(cells.end(), bucket.begin() + cell0[vert[at]], bucket.begin() + cell0[vert[at] + 1]);
        std::sort(cells.begin(), cells.end());
        // (one vertex with more cells than a patch takes: several patches)
        for (size_t c = 0; c < cells.size(); c += max_cells) {
          const size_t n = std::min(cells.size() - c, size_t(max_cells));
          PatchHdr h{};
          h.cell0 = uint32_t(T.cells.size());
          h.node0 = uint32_t(T.nodes.size());
          h.ncells = uint16_t(n);
          T.cells.insert(T.cells.end(), cells.begin() + c, cells.begin() + c + n);
          table.clear();
          for (size_t s = 0; s < n; ++s)
            for (int j = 0; j < k; ++j) {
              const uint32_t node = V.cell_nodes[size_t(cells[c + s]) * k + j];
              if (table.insert(node)) T.nodes.push_back(node);
            }
          std::sort(T.nodes.begin() + h.node0, T.nodes.end());
          h.nnodes = uint16_t(T.nodes.size() - h.node0);
          h.nverts = uint16_t(std::lower_bound(T.nodes.begin() + h.node0, T.nodes.end(), uint32_t(m.nv)) -
                              (T.nodes.begin() + h.node0));
          T.max_nodes = std::max(T.max_nodes, int(h.nnodes));
          T.max_verts = std::max(T.max_verts, int(h.nverts));
          T.hdr.push_back(h);
        }
      }
    }
  }, 1);
  std::vector<size_t> h0(nparts + 1, 0), c0(nparts + 1, 0), n0(nparts + 1, 0), k0(nparts + 1, 0);
  for (int64_t i = 0; i < nparts; ++i) {
    h0[i + 1] = h0[i] + parts[i].hdr.size();
    c0[i + 1] = c0[i] + parts[i].cells.size();
    n0[i + 1] = n0[i] + parts[i].nodes.size();
    for (const PatchHdr& h : parts[i].hdr) B->stride = std::max<int>(B->stride, h.ncells);
    B->max_nodes = std::max(B->max_nodes, parts[i].max_nodes);
    B->max_verts = std::max(B->max_verts, parts[i].max_verts);
  }
  B->stride |= 1;
  B->npatches = int64_t(h0[nparts]);
  // how many patches hold each node; the shared ones' partial slots, filled in
  // patch order
  std::vector<uint32_t> slot(size_t(V.nnodes), 0);
  for (const Part& T : parts)
    for (uint32_t n : T.nodes) slot[n]++;
  B->shared_ptr.push_back(0);
  uint64_t acc = 0;
  for (int64_t n = 0; n < V.nnodes; ++n) {
    const uint32_t c = slot[n];
    slot[n] = c > 1 ? uint32_t(acc) | kPatchPartial : 0u;
    if (c != 1) {  // (c = 0, a vertex of no cell: an empty sum)
      acc += c;
      if (acc >= kPatchPartial) fail(DB2_ERR_UNSUPPORTED, "too many partial sums");
      B->shared.push_back(uint32_t(n));
      B->shared_ptr.push_back(uint32_t(acc));
    }
  }
  B->nshared = int64_t(B->shared.size());
  B->npartial = int64_t(acc);
  std::vector<uint32_t> dest(n0[nparts]);
  for (int64_t i = 0; i < nparts; ++i)
    for (size_t s = 0; s < parts[i].nodes.size(); ++s) {
      const uint32_t n = parts[i].nodes[s];
      dest[n0[i] + s] = slot[n] & kPatchPartial ? slot[n]++ : n;
    }
  // pass 2: connectivity and jobs
  parallel_for(nparts, [&](int64_t b, int64_t e) {
    std::vector<uint32_t> ptr, order;
    std::vector<uint16_t> list, codes;
    std::vector<PatchGroup> groups;
    std::vector<uint32_t> to, fill;
    NodeTable table(size_t(max_cells) * k);
    for (int64_t i = b; i < e; ++i) {
      Part& T = parts[i];
      T.conn.assign(T.cells.size() * kc, 0);
      for (PatchHdr& h : T.hdr) {
        const uint32_t* nodes = T.nodes.data() + h.node0;
        uint16_t* conn = T.conn.data() + size_t(h.cell0) * kc;
        ptr.assign(size_t(h.nnodes) + 1, 0);
        table.clear();
        for (int n = 0; n < h.nnodes; ++n) {
          table.insert(nodes[n]);
          table.val[table.find(nodes[n])] = uint32_t(n);
        }
        for (int c = 0; c < h.ncells; ++c) {
          const uint32_t* cn = &V.cell_nodes[size_t(T.cells[h.cell0 + c]) * k];
          for (int j = 0; j < k; ++j) {
            const uint16_t ln = uint16_t(table.val[table.find(cn[j])]);
            conn[size_t(c) * kc + j] = uint16_t(8 * ln);
            ptr[ln + 1]++;
          }
        }
        for (int n = 0; n < h.nnodes; ++n) ptr[n + 1] += ptr[n];
        list.resize(ptr[h.nnodes]);
        {
          fill.assign(ptr.begin(), ptr.end() - 1);
          for (int c = 0; c < h.ncells; ++c)
            for (int j = 0; j < k; ++j) list[fill[conn[size_t(c) * kc + j] / 8]++] = uint16_t(8 * (j * B->stride + c));
        }
        // longest sums first, so that a group's lanes finish together
        order.resize(h.nnodes);
        std::iota(order.begin(), order.end(), 0u);
        std::stable_sort(order.begin(), order.end(),
                         [&](uint32_t a, uint32_t c) { return ptr[a + 1] - ptr[a] > ptr[c + 1] - ptr[c]; });
        groups.clear();
        codes.clear();
        to.clear();
        const uint16_t zero = uint16_t(8 * k * B->stride);
        for (int g = 0; g < h.nnodes; g += 32) {
          const int live = std::min(32, int(h.nnodes) - g);
          const uint32_t width = ptr[order[g] + 1] - ptr[order[g]];
          const size_t at = codes.size();
          groups.push_back(PatchGroup{uint32_t(at), uint16_t(width), uint16_t(live)});
          codes.resize(at + size_t(width) * 32, zero);
          for (int l = 0; l < 32; ++l) {
            to.push_back(l < live ? dest[n0[i] + h.node0 + order[g + l]] : 0u);
            if (l < live)
              for (uint32_t t = ptr[order[g + l]], q = 0; t < ptr[order[g + l] + 1]; ++t, ++q) codes[at + 32 * q + l] = list[t];
          }
        }
        h.ngroups = uint16_t(groups.size());
        h.chunk0 = uint32_t(T.chunks.size() / 16);
        auto put = [&](const void* src, size_t bytes) {
          const size_t a = T.chunks.size();
          T.chunks.resize(a + PatchPlan::pad16(uint32_t(bytes)), 0);
          if (bytes) std::memcpy(&T.chunks[a], src, bytes);
        };
        put(to.data(), to.size() * 4);
        put(groups.data(), groups.size() * sizeof(PatchGroup));
        put(codes.data(), codes.size() * 2);
        h.chunks = uint32_t(T.chunks.size() / 16) - h.chunk0;
        T.max_chunks = std::max<int>(T.max_chunks, int(h.chunks));
      }
    }
  }, 1);
  for (int64_t i = 0; i < nparts; ++i) {
    k0[i + 1] = k0[i] + parts[i].chunks.size();
    B->max_chunks = std::max(B->max_chunks, parts[i].max_chunks);
  }
  if (n0[nparts] >= (size_t(1) << 32) || k0[nparts] / 16 >= (size_t(1) << 32))
    fail(DB2_ERR_UNSUPPORTED, "cell patches too large");
  B->hdr.resize(h0[nparts]);
  B->nodes.resize(n0[nparts]);
  B->conn.resize(c0[nparts] * kc);
  B->chunks.resize(k0[nparts]);
  parallel_for(nparts, [&](int64_t b, int64_t e) {
    for (int64_t i = b; i < e; ++i) {
      Part& T = parts[i];
      for (auto& h : T.hdr) {
        h.cell0 += uint32_t(c0[i]);
        h.node0 += uint32_t(n0[i]);
        h.chunk0 += uint32_t(k0[i] / 16);
      }
      std::copy(T.hdr.begin(), T.hdr.end(), B->hdr.begin() + h0[i]);
      std::copy(T.conn.begin(), T.conn.end(), B->conn.begin() + c0[i] * kc);
      std::copy(T.nodes.begin(), T.nodes.end(), B->nodes.begin() + n0[i]);
      if (!T.chunks.empty()) std::memcpy(B->chunks.data() + k0[i], T.chunks.data(), T.chunks.size());
      T = Part();
    }
  }, 1);
  return B;
}

// Cells of a patch, measured on B200 at two lattices (ms per action): P2 tets
// n=96 0.246 with 330 cells (five 128-thread CTAs an SM) against 0.284 with 384
// (four), 0.40 with 256; vector P2 elasticity n=48 0.089 with 200 (four CTAs of
// 55 KB); P1 tets n=80 0.062 with 512, 0.066 with 768.  The cuts lie between
// lattice planes, so the caps are met in steps: P2 tets n=96 has 324 cells in
// every patch (1620 resident on an SM), n=40 to 90 and 63x70x57 214 to 267 on
// average (1070 to 1340); elasticity n=48 162 (648 resident), n=30 to 47 129 to
// 192 with CTAs of 61 to 65 KB, of which three fit (387 to 576).
// Small meshes are cut into about 600 patches (four for each of 148 SMs), down
// to 64 cells: one patch's latency is the action's.
const PatchPlan& patch_plan(const Pattern& P) {
  std::lock_guard<std::mutex> guard(P.patches_lock);
  if (!P.patches) {
    const int full = P.V->degree == 1 ? 512 : P.bs > 1 ? 200 : 330;
    auto B = make_patches(P, int(std::min<int64_t>(full, std::max<int64_t>(64, P.V->mesh->nc / 592))));
    for (const PatchHdr& h : B->hdr) {  // (a patch's nodes ascend, vertices first)
      std::array<uint32_t, 4> b{1, 0, 1, 0};  // empty
      const uint32_t* n = B->nodes.data() + h.node0;
      const int k = h.nverts;
      if (k > 0) b[0] = n[0], b[1] = n[k - 1];
      if (k < h.nnodes) b[2] = n[k], b[3] = n[h.nnodes - 1];
      B->bounds.push_back(b);
    }
    PlanUpload U;
    auto up = [&](DeviceBuffer& d, auto& v) {
      if (!v.empty()) U.put(d, v.data(), v.size() * sizeof(v[0]));
      std::remove_reference_t<decltype(v)>().swap(v);
    };
    up(B->d_hdr, B->hdr);
    up(B->d_conn, B->conn);
    up(B->d_nodes, B->nodes);
    up(B->d_chunks, B->chunks);
    // (these two stay on the host too, for the row sets)
    if (B->nshared > 0) U.put(B->d_shared, B->shared.data(), B->shared.size() * sizeof(uint32_t));
    U.put(B->d_shared_ptr, B->shared_ptr.data(), B->shared_ptr.size() * sizeof(uint32_t));
    P.patches = std::move(B);
  }
  return *P.patches;
}

const PatchPlan* patch_plan_for_loads(const Pattern& P) {
  {
    std::lock_guard<std::mutex> guard(P.patches_lock);
    if (P.patches_refused) return nullptr;
  }
  try {
    return &patch_plan(P);
  } catch (const Error& e) {
    if (e.code != DB2_ERR_NOMEM && e.code != DB2_ERR_UNSUPPORTED) throw;
  } catch (const std::bad_alloc&) {
  }
  std::lock_guard<std::mutex> guard(P.patches_lock);
  P.patches_refused = true;
  return nullptr;
}

// Work space that stays with a stream costs a call nothing; from the pool it
// put 1.4 to 1.9 us between the kernels of one call and the next (B200:
// elasticity P2 action n=48 84.5 -> 85.8 us, FP32 P2 63x70x57 78.3 -> 80.2).
CallScratch::CallScratch(const Pattern& P, void* stream) : P_(P), stream_(stream) {
  const PatchPlan& B = *P.patches;
  if (stream_is_capturing(stream)) {
    work_ = &B.captured;
  } else if (const unsigned long long id = stream_id(stream)) {
    std::lock_guard<std::mutex> guard(P.patches_lock);
    for (auto& w : B.works)
      if (w->stream_id == id) work_ = w.get();
    if (!work_ && B.works.size() < PatchPlan::kStreams) {
      B.works.push_back(std::make_unique<PatchPlan::Work>());
      work_ = B.works.back().get();
      work_->stream_id = id;
    }
  }
  if (work_) busy_ = std::unique_lock<std::mutex>(work_->busy);
}

CallScratch::~CallScratch() {
  for (void* p : taken_) P_.patches->scratch.give(p, stream_);
}

double* CallScratch::take(DeviceBuffer PatchPlan::Work::*which, int64_t n) {
  const size_t bytes = size_t(n) * sizeof(double);
  if (work_) {
    DeviceBuffer& d = work_->*which;
    // (actions and loads of a vector space want different lengths; a captured
    // call's never grows, as only actions are captured)
    if (d.bytes < bytes) {
      PlanUpload scope;
      d.alloc(bytes);
    }
    return d.as<double>();
  }
  taken_.reserve(taken_.size() + 1);
  void* p = P_.patches->scratch.take(bytes, stream_);
  if (p) taken_.push_back(p);
  return static_cast<double*>(p);
}

std::shared_ptr<const PatchPlan::RowSet> row_set(const Pattern& P) {
  const PatchPlan& B = *P.patches;
  const int64_t r0 = P.row_begin, r1 = P.row_end < 0 ? P.V->nnodes : P.row_end;
  if (r0 == 0 && r1 == P.V->nnodes) return nullptr;
  std::lock_guard<std::mutex> guard(P.patches_lock);
  for (const auto& s : B.row_sets)
    if (s->begin == r0 && s->end == r1) return s;
  auto S = std::make_shared<PatchPlan::RowSet>();
  S->begin = r0;
  S->end = r1;
  S->verts = r0 < r1 && r0 < P.V->mesh->nv;
  S->edges = r0 < r1 && r1 > P.V->mesh->nv;
  auto first = [&](int64_t row) {
    return uint32_t(std::lower_bound(B.shared.begin(), B.shared.end(), uint32_t(row)) - B.shared.begin());
  };
  S->shared0 = first(r0);
  S->shared1 = std::max(S->shared0, first(r1));
  S->slot0 = B.shared_ptr[S->shared0];
  S->slot1 = B.shared_ptr[S->shared1];
  std::vector<uint32_t> ids;
  auto meets = [&](uint32_t a, uint32_t b) { return r0 < r1 && a <= b && a < r1 && b >= r0; };
  for (size_t i = 0; i < B.bounds.size(); ++i)
    if (meets(B.bounds[i][0], B.bounds[i][1]) || meets(B.bounds[i][2], B.bounds[i][3])) ids.push_back(uint32_t(i));
  S->npatches = int64_t(ids.size());
  PlanUpload U;
  U.put(S->list, ids.data(), ids.size() * sizeof(uint32_t));
  // (a call in progress on another thread holds the set that goes)
  if (B.row_sets.size() >= PatchPlan::kRowSets) B.row_sets.erase(B.row_sets.begin());
  B.row_sets.push_back(S);
  return S;
}

}  // namespace db2
