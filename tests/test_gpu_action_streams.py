"""Actions on one pattern that overlap: several streams of one thread, several
threads, x that is or partly covers y, and a captured action beside eager ones.
Each equals the lone call bit for bit (the order of additions is fixed)."""
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dolfin_b200 as d2

N = 24


def _forms(kind):
    mesh = d2.UnitCubeMesh(N, N, N)
    if kind == "elas":
        V = d2.VectorFunctionSpace(mesh, "Lagrange", 2)
        u, v = d2.TrialFunction(V), d2.TestFunction(V)
        eps = lambda w: d2.sym(d2.grad(w))
        return V, [d2.inner(2 * d2.Constant(m) * eps(u) + d2.Constant(0.6) * d2.tr(eps(u)) * d2.Identity(3), eps(v)) *
                   d2.dx for m in (0.4, 1.4)]
    V = d2.FunctionSpace(mesh, "Lagrange", 2)
    u, v = d2.TrialFunction(V), d2.TestFunction(V)
    return V, [d2.Constant(c) * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx for c in (1.0, -3.0)]


def _x(V, seed):
    return torch.randn(V.dim(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


@pytest.mark.parametrize("kind", ["scalar", "elas"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_streams_of_one_thread(kind, precision):
    V, forms = _forms(kind)
    # (more streams than the pattern keeps work space for)
    jobs = [(forms[i % 2], d2.Vector(_x(V, i))) for i in range(12)]
    alone = [d2.assemble_action(a, x, precision=precision).tensor().clone() for a, x in jobs]
    streams = [torch.cuda.Stream() for _ in jobs]
    outs = [[d2.Vector(n=V.dim()) for _ in range(6)] for _ in jobs]
    torch.cuda.synchronize()
    for r in range(6):
        for s, (a, x), out in zip(streams, jobs, outs):
            with torch.cuda.stream(s):
                d2.assemble_action(a, x, out[r], precision=precision)
    torch.cuda.synchronize()
    for ref, out in zip(alone, outs):
        assert all(torch.equal(y.tensor(), ref) for y in out)


def test_threads_with_x_as_y():
    V, forms = _forms("scalar")
    d2.assemble(forms[0])  # the pattern is resident, the patches are not built
    got = {}
    streams = [torch.cuda.Stream() for _ in range(4)]

    def work(i):
        # threads 0 and 1 share a stream
        with torch.cuda.stream(streams[max(i, 1)]):
            for r in range(6):
                y = d2.Vector(_x(V, 10 * i + r))
                d2.assemble_action(forms[i % 2], y, y)
                got[i, r] = y.tensor()
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (i, r), y in got.items():
        assert torch.equal(y, d2.assemble_action(forms[i % 2], d2.Vector(_x(V, 10 * i + r))).tensor())
    assert len(got) == 24


@pytest.mark.parametrize("shift", [1, -3, 1000])
def test_x_partly_over_y(shift):
    V, forms = _forms("scalar")
    n = V.dim()
    buf = torch.empty(n + 2000, dtype=torch.float64, device="cuda")
    x, y = buf[1000:1000 + n], buf[1000 + shift:1000 + shift + n]
    x.copy_(_x(V, 5))
    ref = d2.assemble_action(forms[0], d2.Vector(x.clone())).tensor()
    d2.assemble_action(forms[0], d2.Vector(x), d2.Vector(y))
    assert torch.equal(y, ref)


def test_captured_action_beside_eager_ones():
    V, forms = _forms("scalar")
    x, z = d2.Vector(_x(V, 1)), d2.Vector(_x(V, 2))
    rx, rz = (d2.assemble_action(forms[0], w).tensor().clone() for w in (x, z))
    y, yz, xy = d2.Vector(n=V.dim()), [d2.Vector(n=V.dim()) for _ in range(6)], d2.Vector(n=V.dim())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        d2.assemble_action(forms[0], x, y)
        xy.tensor().copy_(x.tensor())
        d2.assemble_action(forms[0], xy, xy)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for out in yz:
        g.replay()
        with torch.cuda.stream(s):
            d2.assemble_action(forms[0], z, out)
    torch.cuda.synchronize()
    assert torch.equal(y.tensor(), rx) and torch.equal(xy.tensor(), rx)
    assert all(torch.equal(out.tensor(), rz) for out in yz)
