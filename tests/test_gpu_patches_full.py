"""Actions over patches of their full size: threads that take several cells,
plan data sent ahead to L2, more patches than fit the GPU at once.  Against the
assembled matrix times x: |y - A x| <= tol sum_j |A_ij x_j| with tol = 1e-12
(FP64: a row takes at most a few hundred roundings of 1.1e-16) and 1e-6 (FP32
element actions)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import synthetic

TOL = {"fp64": 1e-12, "fp32": 1e-6}


@pytest.mark.parametrize("dims,deg,kind", [
    ((41, 37, 45), 1, "kappa"), ((41, 37, 45), 1, "const"), ((61, 57, 59), 1, "kappa"),
    ((30, 31, 29), 2, "kappa"), ((30, 31, 29), 2, "const"),
    ((400, 300), 1, "kappa"), ((400, 300), 1, "const"), ((633, 500), 1, "kappa"),
    ((400, 300), 2, "kappa"), ((400, 300), 2, "const"),
    ((41, 37, 45), 1, "elas"), ((30, 31, 29), 2, "elas")])
def test_action_over_full_patches(dims, deg, kind):
    mesh = d2.UnitCubeMesh(*dims) if len(dims) == 3 else d2.UnitSquareMesh(*dims)
    mesh.set_coordinates(synthetic.jitter_interior(mesh.coordinates(), max(dims), 0.15, 31))
    V = d2.FunctionSpace(mesh, "Lagrange", deg, value_size=3 if kind == "elas" else 1)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    if kind == "elas":
        eps = lambda w: d2.sym(d2.grad(w))
        a = d2.inner(2 * d2.Constant(0.4) * eps(u) + d2.Constant(0.7) * d2.tr(eps(u)) * d2.Identity(3), eps(v)) * d2.dx
    elif kind == "const":
        a = d2.Constant(1.7) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    else:
        k = d2.Function(d2.FunctionSpace(mesh, "Lagrange", 1), synthetic.uniform_field(mesh.num_vertices(), 0.5, 2.0, 32))
        a = k * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    rp, cols, vals = d2.assemble(a).data_device()
    x = torch.randn(V.dim(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(33))
    csr = lambda w: torch.sparse_csr_tensor(rp.long(), cols.long(), w, size=(V.dim(), V.dim()))
    ref, mag = csr(vals) @ x, csr(vals.abs()) @ x.abs()
    for precision, tol in TOL.items():
        y = d2.assemble_action(a, d2.Vector(x), precision=precision).tensor()
        assert bool(((y - ref).abs() <= tol * mag).all())
