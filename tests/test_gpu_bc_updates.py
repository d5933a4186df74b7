"""Dirichlet data that changes between assemblies (a time-dependent boundary
value): arrays of dofs_and_values() written in place, a subclass that computes
them anew, an object that is no DirichletBC, and data that is not one value a
dof.  A and b equal, bit for bit, those of a condition made with the data."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2


@pytest.fixture
def problem():
    V = d2.FunctionSpace(d2.UnitCubeMesh(4, 3, 5), "Lagrange", 2)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    return V, d2.inner(d2.grad(u), d2.grad(v)) * d2.dx, d2.Constant(2.0) * v * d2.dx


def _left(x, on):
    return on and x[0] < 1e-12


def _right(x, on):
    return on and x[0] > 1 - 1e-12


def _same(got, want):
    (A, b), (R, r) = got, want
    assert torch.equal(A.values_tensor(), R.values_tensor()) and torch.equal(b.tensor(), r.tensor())


def test_arrays_written_in_place(problem):
    V, a, L = problem
    bc = d2.DirichletBC(V, 1.0, _left)
    S = d2.SystemAssembler(a, L, bc)
    S.assemble()
    dofs, values = bc.dofs_and_values()
    values[:] = 3.5
    _same(S.assemble(), d2.assemble_system(a, L, d2.DirichletBC(V, 3.5, _left)))
    # the dofs of the right face instead (as many)
    dofs[:] = d2.DirichletBC(V, 3.5, _right).dofs_and_values()[0]
    _same(S.assemble(), d2.assemble_system(a, L, d2.DirichletBC(V, 3.5, _right)))


def test_subclass_with_data_of_each_call(problem):
    V, a, L = problem

    class Ramp(d2.DirichletBC):
        def __init__(self, V):
            self.V, self.t = V, 0.0
            self.base = d2.DirichletBC(V, 1.0, _left).dofs_and_values()

        def dofs_and_values(self):
            return self.base[0], self.t * self.base[1]

    bc = Ramp(V)
    S = d2.SystemAssembler(a, L, bc)
    for t in (1.0, 2.0, 2.0, -0.5):
        bc.t = t
        _same(S.assemble(), d2.assemble_system(a, L, d2.DirichletBC(V, t, _left)))


@pytest.mark.parametrize("kind", ["list", "tensor", "scalar", "negative"])
def test_other_objects_and_shapes(problem, kind):
    V, a, L = problem
    dofs, values = d2.DirichletBC(V, 1.5, _left).dofs_and_values()
    data = {"list": (dofs.tolist(), values.tolist()),
            "tensor": (torch.as_tensor(dofs, device="cuda"), torch.as_tensor(values, device="cuda")),
            "scalar": (dofs, np.array(1.5)),
            "negative": (dofs - V.dim(), values)}[kind]

    class Data:
        def dofs_and_values(self):
            return data

    class Sub(d2.DirichletBC):
        def dofs_and_values(self):
            return data

    want = d2.assemble_system(a, L, d2.DirichletBC(V, 1.5, _left))
    for bc in (Data(), Sub(V, 0.0)):
        S = d2.SystemAssembler(a, L, bc)
        _same(S.assemble(), want)
        _same(S.assemble(), want)
