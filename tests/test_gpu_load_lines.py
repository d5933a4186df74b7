"""Load vectors just below and above the sizes from which they run over cell
patches, by element and kind of load, against the oracle (1e-12 of the largest
entry).  The launch count tells which way was taken: one by rows, two over
patches (a P1 load on triangles: two either way)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import synthetic


@pytest.mark.parametrize("dims,deg,kind,patches", [
    ((33, 33, 33), 1, "p1", False), ((34, 34, 34), 1, "p1", True),
    ((57, 57, 57), 1, "const", False), ((58, 58, 58), 1, "const", True),
    ((29, 29, 29), 1, "vector", False), ((30, 30, 30), 1, "vector", True),
    ((17, 17, 17), 2, "const", False), ((18, 18, 18), 2, "const", True),
    ((14, 14, 14), 2, "vector", False), ((15, 15, 15), 2, "vector", True),
    ((752, 752), 1, "p1", None), ((753, 753), 1, "p1", None), ((900, 850), 1, "const", False),
    ((547, 547), 1, "vector", False), ((548, 548), 1, "vector", True),
    ((474, 474), 2, "const", False), ((475, 475), 2, "const", True),
    ((353, 353), 2, "vector", False), ((354, 354), 2, "vector", True)])
def test_both_sides_of_the_load_lines(orc, dims, deg, kind, patches):
    tdim = len(dims)
    om = orc.unit_cube_mesh(*dims) if tdim == 3 else orc.unit_square_mesh(*dims)
    om.coords = synthetic.jitter_interior(om.coords, max(dims), 0.15, 3)
    mesh = d2.Mesh(om.coords, om.cells)
    vs = tdim if kind == "vector" else 1
    V = d2.FunctionSpace(mesh, "Lagrange", deg, value_size=vs)
    v = d2.TestFunction(V)
    od, N = orc.dofmap(om, deg, vs)
    if kind == "p1":
        fv = synthetic.uniform_field(om.nv, -1.0, 1.0, 11)
        L = d2.Function(d2.FunctionSpace(mesh, "Lagrange", 1), fv) * v * d2.dx
        ref = orc.assemble_vector(orc.form(orc.LOAD, tdim, deg, 1, coeff=orc.COEFF_P1), om, od, N, w=fv)
    else:
        c = (-2.5,) if vs == 1 else (0.5, 0.0, -1.5)[:tdim] if tdim == 3 else (0.5, -1.5)
        L = d2.Constant(c[0]) * v * d2.dx if vs == 1 else d2.inner(d2.Constant(c), v) * d2.dx
        ref = orc.assemble_vector(orc.form(orc.LOAD, tdim, deg, vs, coeff=orc.COEFF_CONST, c=c), om, od, N)
    b = d2.assemble(L)
    before = d2.kernel_launches()
    d2.assemble(L, tensor=b)
    launches = d2.kernel_launches() - before
    assert patches is None or launches == (2 if patches else 1)
    assert np.max(np.abs(b.get_local() - ref)) <= 1e-12 * np.max(np.abs(ref))
