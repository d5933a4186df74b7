"""Assemblies by tile classes (several launches on side streams), at sizes just
above those that one launch takes: the join to the caller's stream, a
kappa-weighted load, Dirichlet data of elasticity, accumulation, another launch
shape, row ranges and row blocks.  The launch count of each tells that it ran
by classes.  Against the oracle: 1e-12 of the row's (b: the vector's) largest
entry in FP64, 1e-6 in FP32; otherwise bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import shard, synthetic
from dolfin_b200.autodiff import AssembleDiffusion


def _launches(f):
    before = d2.kernel_launches()
    out = f()
    return out, d2.kernel_launches() - before


def _poisson(n, deg):
    mesh = d2.UnitCubeMesh(n, n, n)
    mesh.set_coordinates(synthetic.jitter_interior(mesh.coordinates(), n, 0.15, 21))
    V, W = d2.FunctionSpace(mesh, "Lagrange", deg), d2.FunctionSpace(mesh, "Lagrange", 1)
    nv = mesh.num_vertices()
    kappa = d2.Function(W, synthetic.uniform_field(nv, 0.5, 2.0, 22))
    f = d2.Function(W, synthetic.uniform_field(nv, -1.0, 1.0, 23))
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    return V, kappa * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, f * v * d2.dx


def _elasticity(n, deg):
    mesh = d2.UnitCubeMesh(n, n, n)
    mesh.set_coordinates(synthetic.jitter_interior(mesh.coordinates(), n, 0.15, 24))
    V = d2.VectorFunctionSpace(mesh, "Lagrange", deg)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    eps = lambda w: d2.sym(d2.grad(w))
    a = d2.inner(2 * d2.Constant(0.7) * eps(u) + d2.Constant(1.3) * d2.tr(eps(u)) * d2.Identity(3), eps(v)) * d2.dx
    return V, a, d2.inner(d2.Constant((0.0, 0.5, -1.0)), v) * d2.dx


def _errors(A, b, ref, bref):
    rp = A.pattern.csr_host()[0]
    scale = np.repeat(np.maximum.reduceat(np.abs(ref), rp[:-1]), np.diff(rp))
    return (np.max(np.abs(A.values_tensor().cpu().numpy() - ref) / scale),
            np.max(np.abs(b.get_local() - bref)) / np.max(np.abs(bref)))


def test_join_to_the_callers_stream():
    V, a, L = _poisson(32, 2)
    S = d2.SystemAssembler(a, L)
    (A0, b0), launches = _launches(S.assemble)
    assert launches >= 3  # packing and two classes at least
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        A1, b1 = S.assemble()
        vals, b = A1.values_tensor().clone(), b1.tensor().clone()  # no host synchronisation before
    torch.cuda.synchronize()
    assert torch.equal(vals, A0.values_tensor()) and torch.equal(b, b0.tensor())


@pytest.mark.parametrize("deg,n", [(1, 40), (2, 30)])
def test_kappa_weighted_load(orc, deg, n):
    mesh = d2.UnitCubeMesh(n, n, n)
    om = orc.unit_cube_mesh(n, n, n)
    V = d2.FunctionSpace(mesh, "Lagrange", deg)
    kv, fv = synthetic.lognormal_field(om.nv, 0.5, 300), synthetic.uniform_field(om.nv, -1.0, 1.0, 301)
    V.pattern().csr_device()
    (vals, b), launches = _launches(lambda: AssembleDiffusion.apply(
        torch.as_tensor(kv, device="cuda"), V, torch.as_tensor(fv, device="cuda"), True, "fp64"))
    assert launches >= (3 if deg == 2 else 2)
    od, N = orc.dofmap(om, deg, 1)
    rp, cols = V.pattern().csr_host()
    ref = orc.assemble_matrix(orc.form(orc.DIFFUSION, 3, deg, 1, coeff=orc.COEFF_P1), om, od, od, rp, cols, w=kv)
    bref = orc.assemble_vector(orc.form(orc.LOAD, 3, deg, 1, coeff=orc.COEFF_P1_TIMES_P1), om, od, N, w=kv, w2=fv)
    scale = np.repeat(np.maximum.reduceat(np.abs(ref), rp[:-1]), np.diff(rp))
    assert np.max(np.abs(vals.cpu().numpy() - ref) / scale) <= 1e-12
    assert np.max(np.abs(b.cpu().numpy() - bref)) <= 1e-12 * np.max(np.abs(bref))


@pytest.mark.parametrize("precision,n,tol", [("fp64", 15, 1e-12), ("fp32", 18, 1e-6)])
def test_elasticity_with_dirichlet_data(orc, precision, n, tol):
    V, a, L = _elasticity(n, 2)
    bc = d2.DirichletBC(V, (0.1, 0.0, -0.2), lambda p, on: on and p[0] < 1e-12)
    S = d2.SystemAssembler(a, L, bc, precision)
    S.assemble()
    (A, b), launches = _launches(S.assemble)
    assert launches >= 2
    om = orc.unit_cube_mesh(n, n, n)
    om.coords = V.mesh().coordinates()
    od, N = orc.dofmap(om, 2, 3)
    rp, cols = A.pattern.csr_host()
    dofs, vals = bc.dofs_and_values()
    order = np.argsort(dofs)
    ref, bref = orc.assemble_system(orc.form(orc.ELASTICITY, 3, 2, 3, mu=0.7, lmbda=1.3),
                                    orc.form(orc.LOAD, 3, 2, 3, coeff=orc.COEFF_CONST, c=(0.0, 0.5, -1.0)), om, od, N,
                                    rp, cols, dofs[order].astype(np.int32), vals[order])
    assert max(_errors(A, b, ref, bref)) <= tol


@pytest.mark.parametrize("precision,n", [("fp64", 30), ("fp32", 38)])
def test_accumulation_and_launch_shape(precision, n):
    V, a, _ = _poisson(n, 2)
    A, launches = _launches(lambda: d2.assemble(a, precision=precision))
    assert launches >= 3
    first = A.values_tensor().clone()
    d2.assemble(a, tensor=A, add_values=True, precision=precision)
    assert torch.allclose(A.values_tensor(), 2 * first, rtol=1e-15, atol=0)
    V.pattern().retile(64, 16 * 1024)
    d2.assemble(a, tensor=A, precision=precision)
    assert torch.equal(A.values_tensor(), first)


@pytest.mark.parametrize("kind", ["poisson", "elasticity"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("bcs", [False, True])
def test_row_ranges_and_blocks(kind, precision, bcs):
    V, a, L = _poisson(38, 2) if kind == "poisson" else _elasticity(19, 2)
    vs = V.value_size()
    bc = d2.DirichletBC(V, 0.25 if vs == 1 else (0.1, 0.0, -0.2), lambda p, on: on and p[0] < 1e-12) if bcs else None
    S = d2.SystemAssembler(a, L, bc, precision)
    A, b = S.assemble()
    P = A.pattern
    _, launches = _launches(lambda: S.assemble(A, b))
    assert launches >= 2
    rv, rb = A.values_tensor().clone(), b.tensor().clone()
    nn = V.dim() // vs
    cuts = shard.row_partition(P.plan()["inc_ptr"], 3)
    rp = torch.as_tensor(P.csr_host()[0].astype(np.int64), device="cuda")
    A.values_tensor().fill_(float("nan"))
    b.tensor().fill_(float("nan"))
    try:
        for r in range(3):
            P.set_row_range(int(cuts[r]), int(cuts[r + 1]))
            S.assemble(A, b)
        assert torch.equal(A.values_tensor(), rv) and torch.equal(b.tensor(), rb)
        for r in range(3):
            blk = shard.RowBlock(V, int(cuts[r]), int(cuts[r + 1]))
            vals, bb = blk.assemble_system(a, L, bc, precision=precision)
            want = [rv[rp[c * nn + int(cuts[r])]:rp[c * nn + int(cuts[r + 1])]] for c in range(vs)]
            assert torch.equal(vals, torch.cat(want))
            assert torch.equal(bb, rb[torch.as_tensor(blk.dofs(), device="cuda")])
    finally:
        P.set_row_range(0, nn)
