"""Cell patches on the host (csrc/patch_plan.cpp), by a program linked to the
engine that stands in for its device calls: meshes with coordinates that are no
numbers, plans that there is no memory for, and the patches of row ranges."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC, LIB = os.path.join(ROOT, "dolfin_b200", "csrc"), os.path.join(ROOT, "dolfin_b200", "_lib")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include <new>
#include "internal.h"
using namespace db2;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""


def _run(tmp_path, body):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None or not os.path.exists(os.path.join(LIB, "libdolfin_b200.so")):
        pytest.skip("needs a C++ compiler and the built engine")
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(PRELUDE + body)
    cuda = os.path.join(CUDA, "lib64")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-rdynamic", "-I", CSRC, str(src), "-o", str(exe), "-L", LIB,
                    "-ldolfin_b200", f"-Wl,-rpath,{LIB}", "-L", cuda, "-lcudart", f"-Wl,-rpath,{cuda}"], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr


def test_coordinates_that_are_no_numbers(tmp_path):
    """The patches are those of the mesh with zeros in their place."""
    _run(tmp_path, r"""
int main() {
  const double bad[] = {std::nan(""), std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity()};
  for (int dim : {2, 3}) {
    std::unique_ptr<PatchPlan> plan[2];
    for (int zero : {0, 1}) {
      auto m = dim == 3 ? make_unit_cube(14, 12, 13) : make_unit_square(60, 50, 0);
      for (int64_t i = 0; i < m->nv; i += 37)
        for (int r = 0; r < dim; ++r) m->x[i * dim + r] = zero ? 0.0 : bad[(i / 37 + r) % 3];
      auto P = make_pattern(make_space(m, 2, 1), false);
      plan[zero] = make_patches(*P, 64);
    }
    CHECK(plan[0]->npatches == plan[1]->npatches && plan[0]->npartial == plan[1]->npartial);
    CHECK(plan[0]->nodes == plan[1]->nodes && plan[0]->conn == plan[1]->conn && plan[0]->chunks == plan[1]->chunks);
  }
  return 0;
}
""")


# uploads that succeed, fail for want of memory, or fail otherwise
UPLOADS = r"""
static int uploads = 0, failure = DB2_OK;
static std::vector<uint32_t> last;  // what was uploaded last
namespace db2 {
PlanUpload::PlanUpload() {}
PlanUpload::~PlanUpload() {}
void PlanUpload::put(DeviceBuffer&, const void* host, size_t n) {
  ++uploads;
  last.assign(static_cast<const uint32_t*>(host), static_cast<const uint32_t*>(host) + n / 4);
  if (failure != DB2_OK) fail(failure, "stand-in");
}
}  // namespace db2
static std::shared_ptr<Pattern> pattern() { return make_pattern(make_space(make_unit_cube(6, 5, 4), 2, 1), false); }
"""


def test_patches_that_cannot_be_built(tmp_path):
    """A load vector's plan that failed for want of memory, or lies beyond the
    plan's limits, is not tried again; another failure is an error each time;
    an action tries, and fails, each time."""
    _run(tmp_path, UPLOADS + r"""
int main() {
  for (int code : {DB2_ERR_NOMEM, DB2_ERR_UNSUPPORTED}) {
    auto P = pattern();
    failure = code;
    uploads = 0;
    CHECK(patch_plan_for_loads(*P) == nullptr && uploads == 1);
    CHECK(patch_plan_for_loads(*P) == nullptr && uploads == 1);
    int caught = 0;
    try { patch_plan(*P); } catch (const Error& e) { caught = e.code; }
    CHECK(caught == code && uploads == 2);
    failure = DB2_OK;
    patch_plan(*P);
    CHECK(patch_plan_for_loads(*P) == nullptr);
  }
  auto P = pattern();
  failure = DB2_ERR_CUDA;
  for (int i = 0; i < 2; ++i) {
    int caught = 0;
    try { patch_plan_for_loads(*P); } catch (const Error& e) { caught = e.code; }
    CHECK(caught == DB2_ERR_CUDA);
  }
  failure = DB2_OK;
  CHECK(patch_plan_for_loads(*P) == &patch_plan(*P));
  return 0;
}
""")


def test_row_sets(tmp_path):
    """A row range's patches, shared nodes and partial slots are those that its
    rows meet, by the plan; a range that comes back (ranges of several ranks in
    turn) is not listed again."""
    _run(tmp_path, UPLOADS + r"""
int main() {
  auto P = pattern();
  patch_plan(*P);
  auto B = make_patches(*P, 64);  // what patch_plan builds for a mesh of 720 cells
  const int64_t nn = P->V->nnodes, nv = P->V->mesh->nv;
  CHECK(row_set(*P) == nullptr && B->npatches > 8);
  const int64_t cuts[][2] = {{0, 0}, {0, nv}, {nv, nn}, {3, 40}, {nv - 5, nv + 7}, {nn - 1, nn}, {0, nn - 1}, {nn, nn}};
  for (auto& c : cuts) {
    P->row_begin = c[0];
    P->row_end = c[1] == nn ? -1 : c[1];
    last.clear();
    auto S = row_set(*P);
    auto in = [&](uint32_t n) { return n >= c[0] && n < c[1]; };
    CHECK(S && S->npatches == int64_t(last.size()));
    size_t at = 0;
    for (int64_t i = 0; i < B->npatches; ++i) {
      bool meets = false;
      for (int j = 0; j < B->hdr[i].nnodes; ++j) meets |= in(B->nodes[B->hdr[i].node0 + j]);
      const bool listed = at < last.size() && last[at] == i;
      CHECK(listed || !meets);
      at += listed;
    }
    CHECK(at == last.size());
    for (size_t i = 0; i < B->shared.size(); ++i) CHECK(in(B->shared[i]) == (i >= S->shared0 && i < S->shared1));
    CHECK(S->slot0 == B->shared_ptr[S->shared0] && S->slot1 == B->shared_ptr[S->shared1]);
    CHECK(S->verts == (c[0] < c[1] && c[0] < nv) && S->edges == (c[0] < c[1] && c[1] > nv));
  }
  const int before = uploads;
  for (int turn = 0; turn < 3; ++turn)
    for (auto& c : cuts) {
      P->row_begin = c[0];
      P->row_end = c[1] == nn ? -1 : c[1];
      CHECK(row_set(*P)->begin == c[0]);
    }
  CHECK(uploads == before);
  for (int64_t i = 1; i < 40; ++i) {  // more than are kept
    P->row_begin = i;
    CHECK(row_set(*P)->begin == i);
  }
  CHECK(P->patches->row_sets.size() == PatchPlan::kRowSets);
  return 0;
}
""")
