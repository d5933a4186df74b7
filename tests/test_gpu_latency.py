"""Assembly on both sides of the size where it changes from one latency-bound
launch to the tile classes: P2 triangles n = 288 and 289 (1.0 million
incidences), P1 tetrahedra n = 38 and 39 (1.4 million), with and without
Dirichlet data, each entry against the oracle (1e-12 of the row's largest entry
in FP64, 1e-6 in FP32); FP32 P2 tetrahedra n = 36 and 37 (3 million) against
FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import synthetic


@pytest.mark.parametrize("tdim,deg,n", [(2, 2, 288), (2, 2, 289), (3, 1, 38), (3, 1, 39)])
@pytest.mark.parametrize("bcs", [False, True])
def test_both_sides_of_the_latency_line(orc, tdim, deg, n, bcs):
    om = orc.unit_square_mesh(n, n) if tdim == 2 else orc.unit_cube_mesh(n, n, n)
    om.coords = synthetic.jitter_interior(om.coords, n, 0.15, 3)
    mesh = d2.Mesh(om.coords, om.cells)
    V = d2.FunctionSpace(mesh, "Lagrange", deg)
    W = d2.FunctionSpace(mesh, "Lagrange", 1)
    kv = synthetic.uniform_field(om.nv, 0.5, 2.0, 4)
    fv = synthetic.uniform_field(om.nv, -1.0, 1.0, 5)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    a = d2.Function(W, kv) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    L = d2.Function(W, fv) * v * d2.dx
    bc = d2.DirichletBC(V, 0.25, lambda p, on: on and p[0] < 1e-12) if bcs else None
    fa = orc.form(orc.DIFFUSION, tdim, deg, 1, coeff=orc.COEFF_P1)
    fL = orc.form(orc.LOAD, tdim, deg, 1, coeff=orc.COEFF_P1)
    od, N = orc.dofmap(om, deg, 1)
    rp, cols = V.pattern().csr_host()
    if bcs:
        dofs, vals = bc.dofs_and_values()
        order = np.argsort(dofs)
        ref, bref = orc.assemble_system(fa, fL, om, od, N, rp, cols, dofs[order].astype(np.int32), vals[order],
                                        wa=kv, wL=fv)
    else:
        ref = orc.assemble_matrix(fa, om, od, od, rp, cols, w=kv)
        bref = orc.assemble_vector(fL, om, od, N, w=fv)
    scale = np.repeat(np.maximum.reduceat(np.abs(ref), rp[:-1]), np.diff(rp))
    for precision, tol in (("fp64", 1e-12), ("fp32", 1e-6)):
        A, b = d2.assemble_system(a, L, bc, precision=precision)
        assert np.max(np.abs(A.values_tensor().cpu().numpy() - ref) / scale) <= tol
        assert np.max(np.abs(b.get_local() - bref)) / np.max(np.abs(bref)) <= tol


@pytest.mark.parametrize("n", [36, 37])
def test_fp32_line_of_p2_tetrahedra(n):
    mesh = d2.UnitCubeMesh(n, n, n)
    mesh.set_coordinates(synthetic.jitter_interior(mesh.coordinates(), n, 0.15, 3))
    V = d2.FunctionSpace(mesh, "Lagrange", 2)
    W = d2.FunctionSpace(mesh, "Lagrange", 1)
    kappa = d2.Function(W, synthetic.uniform_field(mesh.num_vertices(), 0.5, 2.0, 4))
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    a = kappa * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    v64, v32 = d2.assemble(a).values_tensor(), d2.assemble(a, precision="fp32").values_tensor()
    assert not torch.equal(v64, v32)
    rows = V.pattern().csr_device()[0].long()
    row = torch.repeat_interleave(torch.arange(V.dim(), device="cuda"), rows[1:] - rows[:-1])
    scale = torch.zeros(V.dim(), dtype=torch.float64, device="cuda").scatter_reduce_(0, row, v64.abs(), "amax")
    assert float(((v32 - v64).abs() / scale[row]).max()) <= 1e-6
