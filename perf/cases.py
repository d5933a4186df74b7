"""Performance cases of the assembly engine: the calls a finite element program
makes in its loops, through the package's public entry points.

A program builds its mesh, spaces and forms once, makes a first pass (which
creates the matrix and makes the pattern resident on the GPU) and then
assembles, applies or differentiates again and again: a nonlinear or time
loop, a Krylov solver, an optimisation over a coefficient.  ``prepare`` is
that program up to its loop, ``run`` one pass of the loop.

Meshes are the unit cube (six tetrahedra per box) and the unit square, with
interior vertices jittered, as in the package's workloads and tests; the
coefficient kappa is a P1 field in [0.5, 2] (exp of a normal field for the
gradient), the load a P1 field in [-1, 1] or a constant body force.
"""
import numpy as np
import torch

import dolfin_b200 as d2
from dolfin_b200.autodiff import AssembleDiffusion
from dolfin_b200.batch import BatchAssembler

# Elasticity constants: E = 1, nu = 0.3.
MU, LMBDA = 1.0 / 2.6, 0.3 / (1.3 * 0.4)


def listed():
    def c(name, kind, degree, nx, ny, nz, precision="fp64", bcs=False):
        return dict(name=name, kind=kind, degree=degree, nx=nx, ny=ny, nz=nz, precision=precision, bcs=bcs)

    return [
        # A small problem assembled again and again (a time step of a coarse
        # model, a test): the latency of one call counts.
        c("poisson_p1_6x5x7", "poisson_system", 1, 6, 5, 7),
        # The plain Poisson system on a mid-size mesh, 196,608 cells.
        c("poisson_p1_32", "poisson_system", 1, 32, 32, 32),
        # Quadratic Poisson on a large single mesh, 5,308,416 cells.
        c("poisson_p2_96", "poisson_system", 2, 96, 96, 96),
        # The same with the FP32 contraction, on a ragged box.
        c("poisson_p2_fp32_41x37x45", "poisson_system", 2, 41, 37, 45, "fp32"),
        # Boundary value problem as most programs state it: Dirichlet data on
        # the whole boundary.
        c("poisson_p2_dirichlet_23x19x21", "poisson_system", 2, 23, 19, 21, "fp64", True),
        # Linear elasticity with quadratic elements, 2,738,019 unknowns.
        c("elasticity_p2_48", "elasticity_system", 2, 48, 48, 48),
        # One Krylov iteration's operator without a matrix: elasticity in
        # FP64, quadratic Poisson with FP32 element actions.
        c("elasticity_p2_action_48", "elasticity_action", 2, 48, 48, 48),
        c("poisson_p2_action_96", "poisson_action", 2, 96, 96, 96),
        c("poisson_p2_action_fp32_63x70x57", "poisson_action", 2, 63, 70, 57, "fp32"),
        # One step of an optimisation over the coefficient: A(kappa), b(kappa)
        # and the gradient of a functional of both.
        c("poisson_p1_gradient_64", "poisson_gradient", 1, 64, 64, 64),
        # Many independent triangle meshes of uneven size and mixed degree in
        # one launch (nx: smallest n, ny: largest n, nz: how many).
        c("batch_64_squares", "batch", 0, 8, 256, 64),
        # A time loop's right-hand side alone, on triangles.
        c("poisson_p2_rhs_square_500x300", "poisson_rhs", 2, 500, 300, 0),
    ]


# The range of box edges that the drawn cases of each kind come from.  A
# degree of 0 draws 1 or 2; the last edge is 0 on triangles.
_RANGES = {
    "poisson_system": (4, 80),
    "elasticity_system": (3, 40),
    "poisson_action": (8, 90),
    "elasticity_action": (4, 48),
    "poisson_gradient": (6, 72),
    "poisson_rhs": (8, 72),
    "poisson_system_square": (16, 640),
    "poisson_action_square": (16, 640),
}


def draw(rng):
    kind = rng.choice(["batch"] + 2 * sorted(_RANGES))
    if kind == "batch":
        lo = rng.randint(5, 12)
        return dict(kind=kind, degree=0, nx=lo, ny=rng.randint(60, 256), nz=rng.randint(16, 64),
                    precision="fp64", bcs=False)
    lo, hi = _RANGES[kind]
    square = kind.endswith("_square")
    n = lo * (hi / lo) ** rng.random()
    e = [max(lo, min(hi, round(n * rng.uniform(0.75, 1.3)))) for _ in range(3)]
    kind = kind.replace("_square", "")
    precision = "fp32" if rng.random() < 0.25 and kind in ("poisson_system", "poisson_action", "elasticity_action") \
        else "fp64"
    bcs = kind == "poisson_system" and precision == "fp64" and not square and n < 24 and rng.random() < 0.5
    return dict(kind=kind, degree=rng.choice([1, 2, 2]), nx=e[0], ny=e[1], nz=0 if square else e[2],
                precision=precision, bcs=bcs)


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _rng(seed, what):
    return np.random.default_rng([int(seed), what])


def _coordinates(nx, ny, nz, seed):
    """Jittered lattice of the unit cube (nz > 0) or square, x fastest."""
    n = [nx, ny, nz] if nz else [nx, ny]
    axes = [np.arange(m + 1) / m for m in n]
    grid = np.meshgrid(*axes[::-1], indexing="ij")
    x = np.stack([g.ravel() for g in grid[::-1]], axis=1)
    inside = np.all((x > 1e-9) & (x < 1 - 1e-9), axis=1)
    h = np.array([1.0 / m for m in n])
    move = _rng(seed, 1).uniform(-1.0, 1.0, x.shape) * h * (0.15 if nz else 0.2)
    x[inside] += move[inside]
    return x


def _kappa(case, nv, seed):
    if case["kind"] == "poisson_gradient":
        return np.exp(_rng(seed, 2).normal(0.0, 0.5, nv))
    return _rng(seed, 2).uniform(0.5, 2.0, nv)


def _load(nv, seed):
    return _rng(seed, 3).uniform(-1.0, 1.0, nv)


def _gpu_normal(n, seed, what):
    g = torch.Generator("cuda").manual_seed(1000 * int(seed) + what)
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def _members(case):
    """(n, degree) of the members of a batch: n log-uniform in [nx, ny]."""
    r = _rng(case["nx"] + 1000 * case["ny"], case["nz"])
    ns = np.rint(np.exp(r.uniform(np.log(case["nx"]), np.log(case["ny"]), case["nz"]))).astype(int)
    return [(int(n), int(d)) for n, d in zip(ns, r.integers(1, 3, case["nz"]))]


def _mesh(nx, ny, nz, seed):
    mesh = d2.UnitCubeMesh(nx, ny, nz) if nz else d2.UnitSquareMesh(nx, ny)
    mesh.set_coordinates(_coordinates(nx, ny, nz, seed))
    return mesh


def _on_gpu(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind, degree = case["kind"], case["degree"]
    if kind == "batch":
        members = []
        for i, (n, deg) in enumerate(_members(case)):
            s = 100000 * int(seed) + i
            mesh = _mesh(n, n, 0, s)
            V = d2.FunctionSpace(mesh, "Lagrange", deg)
            W = V if deg == 1 else d2.FunctionSpace(mesh, "Lagrange", 1)
            members.append((V, d2.Function(W, _kappa(case, mesh.num_vertices(), s))))
        state = dict(case=case, batch=BatchAssembler(members))
        run(state)
        return state
    mesh = _mesh(case["nx"], case["ny"], case["nz"], seed)
    nv = mesh.num_vertices()
    state = dict(case=case, mesh=mesh)
    if kind.startswith("elasticity"):
        V = d2.VectorFunctionSpace(mesh, "Lagrange", degree)
        u, v = d2.TrialFunction(V), d2.TestFunction(V)
        mu, lmbda = d2.Constant(MU), d2.Constant(LMBDA)

        def eps(w):
            return d2.sym(d2.grad(w))

        a = d2.inner(2 * mu * eps(u) + lmbda * d2.tr(eps(u)) * d2.Identity(3), eps(v)) * d2.dx
        L = d2.inner(d2.Constant((0.0, 0.0, -1.0)), v) * d2.dx
    else:
        V = d2.FunctionSpace(mesh, "Lagrange", degree)
        W = V if degree == 1 else d2.FunctionSpace(mesh, "Lagrange", 1)
        u, v = d2.TrialFunction(V), d2.TestFunction(V)
        kappa, f = d2.Function(W, _kappa(case, nv, seed)), d2.Function(W, _load(nv, seed))
        a = kappa * d2.inner(d2.grad(u), d2.grad(v)) * d2.dx
        L = f * v * d2.dx
    state["V"] = V
    if kind.endswith("system"):
        bcs = [d2.DirichletBC(V, 0.25, "on_boundary")] if case["bcs"] else None
        state["assembler"] = d2.SystemAssembler(a, L, bcs, precision=case["precision"])
        state["A"], state["b"] = state["assembler"].assemble()
    elif kind.endswith("action"):
        state["a"] = a
        state["x"] = d2.Vector(_gpu_normal(V.dim(), seed, 5))
        state["y"] = d2.Vector(n=V.dim())
    elif kind == "poisson_gradient":
        state["kappa"] = _on_gpu(_kappa(case, nv, seed)).requires_grad_(True)
        state["f"] = _on_gpu(_load(nv, seed))
        state["gA"] = _gpu_normal(V.pattern().nnz(), seed, 6)
        state["gb"] = _gpu_normal(V.dim(), seed, 7)
    else:
        state["L"] = L
        state["b"] = d2.Vector(n=V.dim())
    run(state)  # the program's first pass, before its loop
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        return [A.values_tensor() for A in state["batch"].assemble(case["precision"])]
    if kind.endswith("system"):
        A, b = state["assembler"].assemble(state["A"], state["b"])
        return [A.values_tensor(), b.tensor()]
    if kind.endswith("action"):
        return d2.assemble_action(state["a"], state["x"], state["y"], precision=case["precision"]).tensor()
    if kind == "poisson_gradient":
        vals, b = AssembleDiffusion.apply(state["kappa"], state["V"], state["f"], True, case["precision"])
        (dkappa,) = torch.autograd.grad((vals, b), state["kappa"], (state["gA"], state["gb"]))
        return [vals.detach(), b.detach(), dkappa]
    return d2.assemble(state["L"], tensor=state["b"]).tensor()


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _counts(nx, ny, nz):
    """(vertices, edges, faces, cells) of the mesh; faces of triangles: the cells."""
    if nz:
        v = (nx + 1) * (ny + 1) * (nz + 1)
        e = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz \
            + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz
        c = 6 * nx * ny * nz
        return v, e, (4 * c + 4 * (nx * ny + ny * nz + nx * nz)) // 2, c
    v, c = (nx + 1) * (ny + 1), 2 * nx * ny
    return v, nx * (ny + 1) + (nx + 1) * ny + nx * ny, c, c


def _sizes(nx, ny, nz, degree):
    """(vertices, cells, nodes, node pairs of the pattern, nodes per cell)."""
    v, e, f, c = _counts(nx, ny, nz)
    d = 3 if nz else 2
    if degree == 1:
        return v, c, v, v + 2 * e, d + 1
    pairs = v + 7 * e + 12 * f + (6 * c if nz else 0)
    return v, c, v + e, pairs, 10 if nz else 6


def work(case):
    kind, degree, nz = case["kind"], case["degree"], case["nz"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for n, deg in _members(case):
            w = work(dict(case, kind="poisson_matrix", degree=deg, nx=n, ny=n, nz=0))
            total = {k: total[k] + w[k] for k in total}
        return total
    d = 3 if nz else 2
    nv, nc, nn, pairs, k = _sizes(case["nx"], case["ny"], nz, degree)
    bs = d if kind.startswith("elasticity") else 1
    mesh = 4.0 * k * nc + 8.0 * d * nv
    fields = 0.0 if bs > 1 else 8.0 * nv  # kappa or f
    geometry = nc * (30.0 * (d - 1) + (d + 1) * (d + 2) * d)
    entries = nc * 8.0 * bs * bs * k * (k + 1) / 2
    if kind in ("poisson_matrix",):
        return {"bytes": mesh + fields + 8.0 * pairs, "flops": geometry + entries}
    if kind.endswith("action"):
        return {"bytes": mesh + fields + 16.0 * bs * nn, "flops": geometry + nc * 2.0 * bs * k * (d + 1) * (d + 2)}
    if kind == "poisson_rhs":
        return {"bytes": mesh + fields + 8.0 * nn, "flops": geometry + nc * 4.0 * k}
    system = mesh + 2 * fields + 8.0 * bs * bs * pairs + 8.0 * bs * nn
    if kind == "poisson_gradient":
        return {"bytes": system + 8.0 * pairs + 8.0 * nn + 8.0 * nv, "flops": 2 * (geometry + entries)}
    return {"bytes": system, "flops": geometry + entries}


# --------------------------------------------------------------------------
# The same values in plain torch, 64 bits
# --------------------------------------------------------------------------
_TET_EDGES = [(2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1)]
_TRI_EDGES = [(1, 2), (0, 2), (0, 1)]


def _cells(nx, ny, nz):
    sx, sxy = nx + 1, (nx + 1) * (ny + 1)
    if nz:
        iz, iy, ix = torch.meshgrid(torch.arange(nz, device="cuda"), torch.arange(ny, device="cuda"),
                                    torch.arange(nx, device="cuda"), indexing="ij")
        v0 = (iz * sxy + iy * sx + ix).reshape(-1, 1, 1)
        o = [0, 1, sx, sx + 1, sxy, sxy + 1, sxy + sx, sxy + sx + 1]
        t = [(0, 1, 3, 7), (0, 1, 5, 7), (0, 4, 5, 7), (0, 2, 3, 7), (0, 4, 6, 7), (0, 2, 6, 7)]
        return (v0 + torch.tensor([[o[a] for a in r] for r in t], device="cuda")).reshape(-1, 4)
    iy, ix = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
    v0 = (iy * sx + ix).reshape(-1, 1, 1)
    return (v0 + torch.tensor([[0, 1, sx + 1], [0, sx, sx + 1]], device="cuda")).reshape(-1, 3)


def _rule(d, n):
    """Points (barycentric) and weights (of a unit-volume simplex) of the
    collapsed Gauss rule with n points an edge, exact to degree 2 n - d."""
    g, w = np.polynomial.legendre.leggauss(n)
    g, w = (g + 1) / 2, w / 2
    pts, wts = [], []
    if d == 2:
        for a, wa in zip(g, w):
            for b, wb in zip(g, w):
                pts.append((a, b * (1 - a)))
                wts.append(2 * wa * wb * (1 - a))
    else:
        for a, wa in zip(g, w):
            for b, wb in zip(g, w):
                for c, wc in zip(g, w):
                    pts.append((a, b * (1 - a), c * (1 - a) * (1 - b)))
                    wts.append(6 * wa * wb * wc * (1 - a) ** 2 * (1 - b))
    return [[1 - sum(p)] + list(p) for p in pts], wts


def _basis(degree, lam, edges):
    """Values and barycentric derivatives of the Lagrange basis at a point."""
    nb = len(lam)
    if degree == 1:
        return list(lam), [[1.0 if a == i else 0.0 for a in range(nb)] for i in range(nb)]
    val = [x * (2 * x - 1) for x in lam] + [4 * lam[p] * lam[q] for p, q in edges]
    der = [[4 * lam[i] - 1 if a == i else 0.0 for a in range(nb)] for i in range(nb)]
    for p, q in edges:
        der.append([4 * lam[q] if a == p else 4 * lam[p] if a == q else 0.0 for a in range(nb)])
    return val, der


class _Problem:
    """Cells, nodes and geometry of one mesh, worked through in blocks of cells."""

    def __init__(self, nx, ny, nz, degree, seed, rule=3):
        self.d, self.degree = (3 if nz else 2), degree
        self.edges = _TET_EDGES if nz else _TRI_EDGES
        self.x = _on_gpu(_coordinates(nx, ny, nz, seed))
        self.nv = self.x.shape[0]
        self.cells = _cells(nx, ny, nz)
        self.nc = self.cells.shape[0]
        self.nodes, self.nn = self.cells, self.nv
        if degree == 2:
            key = torch.stack([self.cells[:, p] * self.nv + self.cells[:, q] for p, q in self.edges], 1)
            uniq, inv = torch.unique(key, return_inverse=True)
            self.nodes = torch.cat([self.cells, self.nv + inv], 1)
            self.nn = self.nv + uniq.numel()
        self.k = self.nodes.shape[1]
        self.points, self.weights = _rule(self.d, rule)

    def blocks(self, n=250000):
        return [(i, min(self.nc, i + n)) for i in range(0, self.nc, n)]

    def geometry(self, lo, hi):
        """grad(lambda_a) (cells, d + 1, d) and volumes of cells [lo, hi)."""
        X = self.x[self.cells[lo:hi]]
        J = (X[:, 1:] - X[:, :1]).transpose(1, 2)
        g = torch.linalg.inv(J)
        vol = torch.linalg.det(J).abs() / (6 if self.d == 3 else 2)
        return torch.cat([-g.sum(1, keepdim=True), g], 1), vol

    def pattern(self):
        """CSR position of each (cell, i, j) node pair, row pointers."""
        keys = torch.empty(self.nc, self.k, self.k, dtype=torch.int64, device="cuda")
        for lo, hi in self.blocks():
            n = self.nodes[lo:hi]
            keys[lo:hi] = n[:, :, None] * self.nn + n[:, None, :]
        uniq, inv = torch.unique(keys, return_inverse=True)
        del keys
        rows = uniq // self.nn
        rp = torch.zeros(self.nn + 1, dtype=torch.int64, device="cuda")
        rp[1:] = torch.cumsum(torch.bincount(rows, minlength=self.nn), 0)
        return inv, rp, rows, uniq - rows * self.nn

    def point_values(self, q, lo, hi, field):
        return self.weights[q] * sum(self.points[q][a] * field[self.cells[lo:hi, a]] for a in range(self.d + 1))

    def stiffness(self, lo, hi, kappa):
        g, vol = self.geometry(lo, hi)
        A = torch.zeros(hi - lo, self.k, self.k, dtype=torch.float64, device="cuda")
        for q in range(len(self.weights)):
            G = torch.einsum("ja,cad->cjd", _on_gpu(_basis(self.degree, self.points[q], self.edges)[1]), g)
            A += (self.point_values(q, lo, hi, kappa) * vol)[:, None, None] * (G @ G.transpose(1, 2))
        return A

    def load(self, lo, hi, f, kappa=None):
        vol = self.geometry(lo, hi)[1]
        b = torch.zeros(hi - lo, self.k, dtype=torch.float64, device="cuda")
        for q in range(len(self.weights)):
            w = self.point_values(q, lo, hi, f) * vol
            if kappa is not None:
                w = w * self.point_values(q, lo, hi, kappa) / self.weights[q]
            b += w[:, None] * _on_gpu(_basis(self.degree, self.points[q], self.edges)[0])
        return b

    def gradients(self, lo, hi):
        """B[c, e, i, j] = int d_c phi_i d_e phi_j."""
        g, vol = self.geometry(lo, hi)
        B = torch.zeros(hi - lo, 3, 3, self.k, self.k, dtype=torch.float64, device="cuda")
        for q in range(len(self.weights)):
            G = torch.einsum("ja,cad->cdj", _on_gpu(_basis(self.degree, self.points[q], self.edges)[1]), g)
            B += (self.weights[q] * vol)[:, None, None, None, None] * G[:, :, None, :, None] * G[:, None, :, None, :]
        return B

    def elasticity(self, lo, hi):
        """A[c, e, i, j] of 2 mu eps(u):eps(v) + lmbda div(u) div(v)."""
        B = self.gradients(lo, hi)
        A = LMBDA * B + MU * B.transpose(1, 2)
        tr = MU * (B[:, 0, 0] + B[:, 1, 1] + B[:, 2, 2])
        for c in range(3):
            A[:, c, c] += tr
        return A


def _scalar_system(P, case, seed):
    kappa, f = _on_gpu(_kappa(case, P.nv, seed)), _on_gpu(_load(P.nv, seed))
    inv, rp, rows, cols = P.pattern()
    vals = torch.zeros(rows.numel(), dtype=torch.float64, device="cuda")
    b = torch.zeros(P.nn, dtype=torch.float64, device="cuda")
    weighted = kappa if case["kind"] == "poisson_gradient" else None
    for lo, hi in P.blocks():
        vals.index_add_(0, inv[lo:hi].reshape(-1), P.stiffness(lo, hi, kappa).reshape(-1))
        b.index_add_(0, P.nodes[lo:hi].reshape(-1), P.load(lo, hi, f, weighted).reshape(-1))
    return vals, b, inv, rows, cols


def _with_dirichlet(P, vals, b, rows, cols, value):
    """Symmetric elimination, one unit of diagonal per incident cell."""
    nb = P.d + 1
    facets = [[a for a in range(nb) if a != s] for s in range(nb)]
    fv = torch.cat([P.cells[:, f] for f in facets])
    key = fv[:, 0]
    for r in range(1, P.d):
        key = key * P.nv + fv[:, r]
    _, inv, count = torch.unique(key, return_inverse=True, return_counts=True)
    once = (count[inv] == 1).reshape(nb, -1)
    flag = torch.zeros(P.nn, dtype=torch.bool, device="cuda")
    for s, f in enumerate(facets):
        local = f + [nb + i for i, (p, q) in enumerate(P.edges) if P.degree == 2 and s not in (p, q)]
        flag[P.nodes[once[s]][:, local].reshape(-1)] = True
    cells = torch.bincount(P.nodes.reshape(-1), minlength=P.nn).to(torch.float64)
    moved = ~flag[rows] & flag[cols]
    b = b.index_add(0, rows[moved], -value * vals[moved])
    b[flag] = value * cells[flag]
    vals = vals * ~(flag[rows] | flag[cols])
    own = flag[rows] & (rows == cols)
    vals[own] = cells[rows[own]]
    return vals, b


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for i, (n, deg) in enumerate(_members(case)):
            s = 100000 * int(seed) + i
            out.append(_scalar_system(_Problem(n, n, 0, deg, s), case, s)[0])
        return out
    # kappa f phi_i of a quadratic basis has degree 4
    P = _Problem(case["nx"], case["ny"], case["nz"], case["degree"], seed, 4 if kind == "poisson_gradient" else 3)
    if kind == "poisson_system":
        vals, b, _, rows, cols = _scalar_system(P, case, seed)
        return list(_with_dirichlet(P, vals, b, rows, cols, 0.25)) if case["bcs"] else [vals, b]
    if kind == "poisson_rhs":
        f = _on_gpu(_load(P.nv, seed))
        b = torch.zeros(P.nn, dtype=torch.float64, device="cuda")
        for lo, hi in P.blocks():
            b.index_add_(0, P.nodes[lo:hi].reshape(-1), P.load(lo, hi, f).reshape(-1))
        return b
    if kind == "poisson_gradient":
        vals, b, inv, _, _ = _scalar_system(P, case, seed)
        f, gA, gb = _on_gpu(_load(P.nv, seed)), _gpu_normal(vals.numel(), seed, 6), _gpu_normal(P.nn, seed, 7)
        dk = torch.zeros(P.nv, dtype=torch.float64, device="cuda")
        for lo, hi in P.blocks():
            g, vol = P.geometry(lo, hi)
            up, ub = gA[inv[lo:hi]], gb[P.nodes[lo:hi]]
            for q, w in enumerate(P.weights):
                phi, der = _basis(P.degree, P.points[q], P.edges)
                G = torch.einsum("ja,cad->cjd", _on_gpu(der), g)
                t = w * (up * (G @ G.transpose(1, 2))).sum((1, 2)) + P.point_values(q, lo, hi, f) * (ub @ _on_gpu(phi))
                for a in range(P.d + 1):
                    dk.index_add_(0, P.cells[lo:hi, a], P.points[q][a] * t * vol)
        return [vals, b, dk]
    if kind == "poisson_action":
        kappa, x = _on_gpu(_kappa(case, P.nv, seed)), _gpu_normal(P.nn, seed, 5)
        y = torch.zeros(P.nn, dtype=torch.float64, device="cuda")
        for lo, hi in P.blocks():
            n = P.nodes[lo:hi]
            y.index_add_(0, n.reshape(-1), (P.stiffness(lo, hi, kappa) @ x[n][:, :, None]).reshape(-1))
        return y
    if kind == "elasticity_action":
        x = _gpu_normal(3 * P.nn, seed, 5).reshape(3, P.nn)
        y = torch.zeros(3, P.nn, dtype=torch.float64, device="cuda")
        for lo, hi in P.blocks(60000):
            n = P.nodes[lo:hi]
            yc = torch.einsum("mceij,emj->cmi", P.elasticity(lo, hi), x[:, n])
            y.index_add_(1, n.reshape(-1), yc.reshape(3, -1))
        return y.reshape(-1)
    # elasticity_system: component-major dofs, row (c, i) holds its blocks e in order
    inv, rp, rows, _ = P.pattern()
    nnz = rows.numel()
    A = torch.zeros(3, 3, nnz, dtype=torch.float64, device="cuda")
    b = torch.zeros(3, P.nn, dtype=torch.float64, device="cuda")
    ones = torch.ones(P.nv, dtype=torch.float64, device="cuda")
    for lo, hi in P.blocks(60000):
        at = inv[lo:hi].reshape(-1)
        A.index_add_(2, at, P.elasticity(lo, hi).permute(1, 2, 0, 3, 4).reshape(3, 3, -1))
        b[2].index_add_(0, P.nodes[lo:hi].reshape(-1), -P.load(lo, hi, ones).reshape(-1))
    length = (rp[1:] - rp[:-1])[rows]
    at = 3 * rp[rows] + torch.arange(nnz, device="cuda") - rp[rows]
    vals = torch.empty(9 * nnz, dtype=torch.float64, device="cuda")
    for c in range(3):
        for e in range(3):
            vals[3 * c * nnz + at + e * length] = A[c, e]
    return [vals, b.reshape(-1)]
