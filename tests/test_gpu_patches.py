"""Matrix-free action and load vector over cell patches.  The action against the
oracle's CSR times x:
one patch and many, patches that share nodes, ragged boxes, permuted vertex
numbering, a vertex of no cell, and an x that is also y.  Row-wise bound:
|y - R x| <= tol sum_j |R_ij x_j| with tol = 1e-12 (FP64: a row takes at most
a few hundred roundings of 1.1e-16) and 1e-6 (FP32 element actions)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2
from dolfin_b200 import synthetic

TOL = {"fp64": 1e-12, "fp32": 1e-6}


def _mesh(orc, dims, permute):
    om = orc.unit_cube_mesh(*dims) if len(dims) == 3 else orc.unit_square_mesh(*dims)
    x = om.coords + np.random.default_rng(7).uniform(-0.1, 0.1, om.coords.shape) / max(dims)
    if permute:
        perm = np.random.default_rng(8).permutation(om.nv)
        xp = np.empty_like(x)
        xp[perm] = x
        cells = np.sort(perm[om.cells.astype(np.int64)], axis=1).astype(np.uint32)
        return orc.Mesh(len(dims), xp, cells)
    return orc.Mesh(len(dims), x, om.cells)


def _form(V, kind, nv):
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    if kind == "elas":
        mu, lm = 0.4, 0.7
        eps = lambda w: d2.sym(d2.grad(w))
        return d2.inner(2 * d2.Constant(mu) * eps(u) + d2.Constant(lm) * d2.tr(eps(u)) * d2.Identity(3),
                        eps(v)) * d2.dx, None, dict(mu=mu, lmbda=lm)
    if kind == "const":
        return d2.Constant(1.7) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, None, dict(c=(1.7,))
    kv = synthetic.uniform_field(nv, 0.5, 2.0, 9)
    W = d2.FunctionSpace(V.mesh(), "Lagrange", 1)
    return d2.Function(W, kv) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, kv, {}


def _oracle_csr(orc, om, deg, kind, kv, kw, V):
    import scipy.sparse as sp
    vs = 3 if kind == "elas" else 1
    od, N = orc.dofmap(om, deg, vs)
    rp, cols = V.pattern().csr_host()
    if kind == "elas":
        f = orc.form(orc.ELASTICITY, 3, deg, 3, **kw)
    else:
        f = orc.form(orc.DIFFUSION, om.coords.shape[1], deg, 1,
                     coeff=orc.COEFF_P1 if kv is not None else orc.COEFF_CONST, c=kw.get("c", (0, 0, 0)))
    ref = orc.assemble_matrix(f, om, od, od, rp, cols, w=kv)
    return sp.csr_matrix((ref, cols, rp), shape=(N, N))


@pytest.mark.parametrize("dims,permute", [((1, 1, 1), False), ((5, 4, 3), False), ((9, 7, 8), False),
                                          ((6, 6, 6), True), ((1, 1), False), ((23, 17), False)])
@pytest.mark.parametrize("deg", [1, 2])
@pytest.mark.parametrize("kind", ["kappa", "const", "elas"])
def test_action_over_patches(orc, dims, permute, deg, kind):
    if kind == "elas" and len(dims) == 2:
        pytest.skip("elasticity is provided on tetrahedra")
    om = _mesh(orc, dims, permute)
    mesh = d2.Mesh(om.coords, om.cells)
    V = d2.FunctionSpace(mesh, "Lagrange", deg, value_size=3 if kind == "elas" else 1)
    a, kv, kw = _form(V, kind, om.nv)
    R = _oracle_csr(orc, om, deg, kind, kv, kw, V)
    x = np.random.default_rng(10).standard_normal(V.dim())
    mag = abs(R) @ np.abs(x)
    for prec, tol in TOL.items():
        xt = d2.Vector(torch.as_tensor(x, device="cuda"))
        y = d2.assemble_action(a, xt, precision=prec).get_local()
        assert np.all(np.abs(y - R @ x) <= tol * mag)
        # x itself as y
        d2.assemble_action(a, xt, xt, precision=prec)
        assert np.array_equal(xt.get_local(), y)


def test_vertex_of_no_cell_gets_zero():
    x = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [5, 5, 5]], float)
    mesh = d2.Mesh(x, np.array([[0, 1, 2, 3]], np.uint32))
    V = d2.FunctionSpace(mesh, "Lagrange", 1)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    y = d2.Vector(torch.full((5,), float("nan"), dtype=torch.float64, device="cuda"))
    one = d2.Vector(torch.arange(5, dtype=torch.float64, device="cuda"))
    d2.assemble_action(d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, one, y)
    got = y.get_local()
    # grad u = (1, 2, 3) on the reference tetrahedron, |T| = 1/6
    assert np.allclose(got, [-1.0, 1 / 6, 2 / 6, 3 / 6, 0.0], rtol=0, atol=1e-15) and got[4] == 0.0


def test_first_action_inside_a_graph_capture():
    """The patches are built on the first action, also when that one is being
    captured; replays see the x of their time."""
    mesh = d2.UnitCubeMesh(4, 4, 4)
    V = d2.FunctionSpace(mesh, "Lagrange", 2)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    a = d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    d2.assemble(a)  # the pattern is resident, the patches are not built
    x = d2.Vector(torch.zeros(V.dim(), dtype=torch.float64, device="cuda"))
    y = d2.Vector(n=V.dim())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        d2.assemble_action(a, x, y)
    xv = torch.randn(V.dim(), dtype=torch.float64, device="cuda")
    x.tensor().copy_(xv)
    g.replay()
    torch.cuda.synchronize()
    ref = d2.assemble_action(a, d2.Vector(xv)).tensor()
    assert torch.equal(y.tensor(), ref)


@pytest.mark.parametrize("dims,deg", [((14, 14, 14), 2), ((15, 15, 15), 2), ((20, 20, 20), 1), ((21, 21, 21), 1),
                                      ((353, 353), 2), ((354, 354), 2)])
@pytest.mark.parametrize("kind", ["p1", "const"])
def test_load_vector_on_both_sides_of_the_patch_line(orc, dims, deg, kind):
    """Tetrahedra change at 200,000 incidences (P2 n = 14 / 15, P1 n = 20 / 21),
    triangles at 1.5 million (P2 n = 353 / 354); each entry against the oracle
    (1e-12 of the largest), accumulation, and row ranges bit for bit."""
    om = _mesh(orc, dims, False)
    mesh = d2.Mesh(om.coords, om.cells)
    V = d2.FunctionSpace(mesh, "Lagrange", deg)
    v = d2.TestFunction(V)
    od, N = orc.dofmap(om, deg, 1)
    if kind == "p1":
        fv = synthetic.uniform_field(om.nv, -1.0, 1.0, 11)
        L = d2.Function(d2.FunctionSpace(mesh, "Lagrange", 1), fv) * v * d2.dx
        ref = orc.assemble_vector(orc.form(orc.LOAD, len(dims), deg, 1, coeff=orc.COEFF_P1), om, od, N, w=fv)
    else:
        L = d2.Constant(-2.5) * v * d2.dx
        ref = orc.assemble_vector(orc.form(orc.LOAD, len(dims), deg, 1, coeff=orc.COEFF_CONST, c=(-2.5,)), om, od, N)
    b = d2.assemble(L)
    got = b.get_local()
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    d2.assemble(L, tensor=b, add_values=True)
    assert np.allclose(b.get_local(), 2 * got, rtol=1e-15, atol=0)
    P = V.pattern()
    part = d2.Vector(torch.full((N,), float("nan"), dtype=torch.float64, device="cuda"))
    try:
        for a, e in ((0, om.nv // 3), (om.nv // 3, N - 5), (N - 5, N)):
            P.set_row_range(a, e)
            d2.assemble(L, tensor=part)
    finally:
        P.set_row_range(0, N)
    assert np.array_equal(part.get_local(), got)


def test_vector_load_over_patches(orc):
    om = _mesh(orc, (15, 15, 15), False)
    mesh = d2.Mesh(om.coords, om.cells)
    V = d2.VectorFunctionSpace(mesh, "Lagrange", 2)
    c = (0.5, 0.0, -1.5)
    b = d2.assemble(d2.inner(d2.Constant(c), d2.TestFunction(V)) * d2.dx)
    od, N = orc.dofmap(om, 2, 3)
    ref = orc.assemble_vector(orc.form(orc.LOAD, 3, 2, 3, coeff=orc.COEFF_CONST, c=c), om, od, N)
    assert np.max(np.abs(b.get_local() - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_load_vectors_on_several_streams_and_under_capture():
    """Calls on one pattern that overlap (four streams) have partial sums of
    their own: each equals the lone call bit for bit.  A captured call sums by
    rows (1e-13 of the largest: ~120 terms a row)."""
    V = d2.FunctionSpace(d2.UnitCubeMesh(24, 24, 24), "Lagrange", 2)
    v = d2.TestFunction(V)
    Ls = [d2.Constant(c) * v * d2.dx for c in (1.0, -3.0, 0.5, 7.0)]
    alone = [d2.assemble(L).get_local() for L in Ls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in Ls]
    outs = [[d2.Vector(n=V.dim()) for _ in range(8)] for _ in Ls]
    torch.cuda.synchronize()
    for r in range(8):
        for s, L, out in zip(streams, Ls, outs):
            with torch.cuda.stream(s):
                d2.assemble(L, tensor=out[r])
    torch.cuda.synchronize()
    for ref, out in zip(alone, outs):
        for b in out:
            assert np.array_equal(b.get_local(), ref)
    b = d2.Vector(n=V.dim())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        d2.assemble(Ls[1], tensor=b)
    g.replay()
    torch.cuda.synchronize()
    assert np.max(np.abs(b.get_local() - alone[1])) <= 1e-13 * np.max(np.abs(alone[1]))
