"""AssembleDiffusion on a pattern that assembles a part of its rows: the others
are zero, also when the range was set through the C entry point; a vertex of
no cell gets b = 0.  The allocator's free blocks are filled with NaN first."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import _capi
from dolfin_b200.autodiff import AssembleDiffusion


def _poison(*sizes):
    held = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for n in sizes for _ in range(4)]
    torch.cuda.synchronize()
    del held


@pytest.mark.parametrize("through", ["python", "c"])
def test_rows_outside_the_range_are_zero(through):
    V = d2.FunctionSpace(d2.UnitCubeMesh(5, 4, 6), "Lagrange", 2)
    nv = V.mesh().num_vertices()
    kappa = torch.linspace(0.5, 2.0, nv, dtype=torch.float64, device="cuda")
    f = torch.linspace(-1.0, 1.0, nv, dtype=torch.float64, device="cuda")
    A, b = AssembleDiffusion.apply(kappa, V, f)
    P = V.pattern()
    rp = P.csr_host()[0]
    a, e, nn = 100, 700, V.dim()
    try:
        if through == "python":
            P.set_row_range(a, e)
        else:
            _capi.call("db2_pattern_set_row_range", P.handle, a, e)
        assert P.has_row_range()
        _poison(P.nnz(), V.dim())
        Ar, br = AssembleDiffusion.apply(kappa, V, f)
    finally:
        P.set_row_range(0, nn)
    assert not P.has_row_range()
    want, wb = torch.zeros_like(A), torch.zeros_like(b)
    want[rp[a]:rp[e]] = A[rp[a]:rp[e]]
    wb[a:e] = b[a:e]
    assert torch.equal(Ar, want) and torch.equal(br, wb)


def test_vertex_of_no_cell():
    x = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [5, 5, 5]], float)
    V = d2.FunctionSpace(d2.Mesh(x, np.array([[0, 1, 2, 3]], np.uint32)), "Lagrange", 1)
    one = torch.ones(5, dtype=torch.float64, device="cuda")
    V.pattern()
    _poison(V.pattern().nnz(), 5)
    A, b = AssembleDiffusion.apply(one, V, one)
    assert torch.isfinite(A).all() and b[4] == 0.0
