"""Outputs that share memory with the coefficient of the call: b, the CSR values
or y over kappa (exactly, or a few doubles off), and over f on triangles, on both
sides of the sizes where the calls change their kernels.  Against the same call
with outputs of its own: 1e-13 of the largest entry (the row sums have the same
terms, at most a few hundred, in another grouping)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2


def _mesh(dims):
    return d2.UnitCubeMesh(*dims) if len(dims) == 3 else d2.UnitSquareMesh(*dims)


def _field(n, seed):
    return 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _over(values, out_len, shift):
    """(view of `values`, view of out_len doubles `shift` doubles behind it) of one array."""
    buf = torch.zeros(max(out_len, values.numel()) + abs(shift) + 8, dtype=torch.float64, device="cuda")
    at = max(0, -shift)
    view = buf[at:at + values.numel()]
    view.copy_(values)
    return view, buf[at + shift:at + shift + out_len]


def _close(got, ref):
    assert float((got - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


@pytest.mark.parametrize("dims", [(9, 8, 7), (40, 40, 40), (30, 20), (360, 350)])
@pytest.mark.parametrize("deg", [1, 2])
@pytest.mark.parametrize("what", ["b over kappa", "b over f", "values over kappa"])
@pytest.mark.parametrize("shift", [0, 4, -4])
def test_system(dims, deg, what, shift):
    if what == "b over f" and len(dims) == 3:
        pytest.skip("f must lie apart from b on tetrahedra")
    mesh = _mesh(dims)
    V, W = d2.FunctionSpace(mesh, "Lagrange", deg), d2.FunctionSpace(mesh, "Lagrange", 1)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    nv, P = mesh.num_vertices(), V.pattern()
    kt, ft = _field(nv, 1), _field(nv, 2)
    vals, b = d2.Matrix(P).values_tensor(), torch.zeros(V.dim(), dtype=torch.float64, device="cuda")

    def assemble(kt, ft, vals, b):
        k, f = d2.Function(W, kt), d2.Function(W, ft)
        S = d2.SystemAssembler(k * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, f * v * d2.dx)
        S.assemble_into(P, vals, b)

    assemble(kt, ft, vals, b)
    rv, rb = vals.clone(), b.clone()
    if what == "b over kappa":
        kt, b = _over(kt, V.dim(), shift)
    elif what == "b over f":
        ft, b = _over(ft, V.dim(), shift)
    else:
        kt, vals = _over(kt, P.nnz(), shift)
    assemble(kt, ft, vals, b)
    _close(vals, rv)
    _close(b, rb)


@pytest.mark.parametrize("dims,deg", [((30, 20), 1), ((30, 20), 2), ((360, 350), 2), ((720, 700), 1)])
@pytest.mark.parametrize("shift", [0, 4, -4])
def test_load_vector_over_f_on_triangles(dims, deg, shift):
    mesh = _mesh(dims)
    V, W = d2.FunctionSpace(mesh, "Lagrange", deg), d2.FunctionSpace(mesh, "Lagrange", 1)
    v = d2.TestFunction(V)
    ft = _field(mesh.num_vertices(), 3)
    ref = d2.assemble(d2.Function(W, ft) * v * d2.dx).tensor().clone()
    ft, b = _over(ft, V.dim(), shift)
    d2.assemble(d2.Function(W, ft) * v * d2.dx, tensor=d2.Vector(b))
    _close(b, ref)


@pytest.mark.parametrize("dims", [(9, 8, 7), (40, 40, 40), (30, 20), (360, 350)])
@pytest.mark.parametrize("deg", [1, 2])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shift", [0, 4, -4])
def test_action_over_kappa(dims, deg, precision, shift):
    mesh = _mesh(dims)
    V, W = d2.FunctionSpace(mesh, "Lagrange", deg), d2.FunctionSpace(mesh, "Lagrange", 1)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    kt, x = _field(mesh.num_vertices(), 4), d2.Vector(_field(V.dim(), 5))
    form = lambda k: d2.Function(W, k) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
    ref = d2.assemble_action(form(kt), x, precision=precision).tensor().clone()
    kt, y = _over(kt, V.dim(), shift)
    d2.assemble_action(form(kt), x, d2.Vector(y), precision=precision)
    assert torch.equal(y, ref)
