"""Workloads that stand for what users of the library run, each through its public
entry points: operator applications (GLL collocation, Gauss points, vector-valued,
on host vectors), the element kernels behind them, and whole solves.

``listed()`` names the representative ones, ``draw(rng)`` gives more of the same
ranges, ``prepare``/``run`` set a workload up and execute one pass, ``work`` counts
the bytes and operations a pass cannot do without, and ``exact`` computes the same
results in 64 bits with plain torch."""
import math

import numpy as np
import torch

import benchmarks_gb300 as mf

# Largest problem exact() solves or applies, in unknowns
SOLVE_LIMIT = 9_000_000


def listed():
    return [
        # 117,649 unknowns: the smallest mesh of the solver studies, bound by launches and latency
        dict(name="apply_q3_small", kind="apply", form="gll", arith="df", p=3, nx=16, ny=16, nz=16),
        # 67.6 M unknowns: the operator benchmark's own mesh
        dict(name="apply_q4_large", kind="apply", form="gll", arith="df", p=4, nx=128, ny=128, nz=64),
        # odd cell counts at a higher degree, 8.1 M unknowns: the middle of the degree x size study
        dict(name="apply_q6_odd", kind="apply", form="gll", arith="df", p=6, nx=33, ny=35, nz=32),
        # the native FP64 arithmetic, on a mesh a preconditioner study would take
        dict(name="apply_q5_fp64", kind="apply", form="gll", arith="fp64", p=5, nx=30, ny=31, nz=29),
        # QGauss(p+1), the form the published BP5 results use
        dict(name="apply_gauss_q4", kind="apply", form="gauss", arith="df", p=4, nx=64, ny=64, nz=32),
        # QGauss(p+2), the BP3 operator
        dict(name="apply_bp3_q5", kind="apply", form="bp3", arith="df", p=5, nx=25, ny=24, nz=23),
        # three components (BK6), 4.2 M nodes
        dict(name="vector_q4", kind="vector", form="gll", arith="df", p=4, nx=40, ny=40, nz=40),
        # a caller with host vectors: the copies are part of the call
        dict(name="host_q4", kind="host", form="gll", arith="df", p=4, nx=64, ny=64, nz=64),
        # the CEED BK3 element kernel on caller-supplied geometry
        dict(name="bk3_q4", kind="bk3", arith="df", p=4, nelmt=100_000),
        # Jacobi-preconditioned CG to 1e-8 on the smallest mesh
        dict(name="cg_q3_small", kind="cg", form="gll", arith="df", p=3, nx=16, ny=16, nz=16, reduce=1e-8),
        # multigrid-preconditioned CG to 1e-10, 8.5 M unknowns
        dict(name="mg_q4", kind="mg", form="gll", arith="df", p=4, nx=64, ny=64, nz=32, reduce=1e-10),
        # many independent problems of mixed degree and size, solved together
        dict(name="batch_mixed", kind="batch", problems=24, mix=2024, reduce=1e-10),
    ]


def draw(rng):
    def cells(p, low, high):
        n = math.exp(rng.uniform(math.log(low), math.log(high))) ** (1 / 3) / p
        f, g = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
        return dict(nx=max(2, round(n * f)), ny=max(2, round(n * g)), nz=max(2, round(n / (f * g))))

    kind = rng.choice(["apply"] * 8 + ["gauss"] * 3 + ["vector"] * 2 + ["host", "seam", "seam", "cg", "mg"])
    p = rng.randint(1, 8)
    if kind == "apply":
        arith = rng.choice(["df", "df", "df", "fp64"])
        return dict(kind="apply", form="gll", arith=arith, p=p, **cells(p, 1e5, 4e7 if arith == "df" else 1e7))
    if kind == "gauss":
        return dict(kind="apply", form=rng.choice(["gauss", "bp3", "helmholtz"]), arith="df", p=p, **cells(p, 1e5, 1e7))
    if kind == "vector":
        return dict(kind="vector", form="gll", arith="df", p=p, **cells(p, 1e5, 5e6))
    if kind == "host":
        return dict(kind="host", form="gll", arith="df", p=p, **cells(p, 1e6, 1.7e7))
    if kind == "seam":
        return dict(kind=rng.choice(["bk1", "bk3", "bk5"]), arith="df", p=p,
                    nelmt=round(math.exp(rng.uniform(math.log(1e5), math.log(1.2e7))) / (p + 1) ** 3))
    p = rng.randint(2, 8)
    if kind == "cg":
        return dict(kind="cg", form="gll", arith="df", p=p, reduce=1e-8, **cells(p, 5e4, 2e5))
    return dict(kind="mg", form="gll", arith="df", p=p, reduce=1e-10, **cells(p, 1e6, 8e6))


# ---- one pass through the library ------------------------------------------
def _mesh(case):
    return mf.BoxMesh(case["nx"], case["ny"], case["nz"], degree=case["p"])


def _uniform(n, g):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _interior(case, v):
    """v with 0 on the Dirichlet boundary."""
    n = [case["p"] * case[d] + 1 for d in ("nz", "ny", "nx")]
    w = torch.zeros(n, dtype=v.dtype, device=v.device)
    w[1:-1, 1:-1, 1:-1] = v.view(n)[1:-1, 1:-1, 1:-1]
    return w.view(-1)


def _element_inputs(case, seed):
    """Geometry and values of independent elements: symmetric positive factors, as of mildly deformed cells."""
    g = _generator(seed)
    n = case["p"] + 1
    nq, e = (n if case["kind"] == "bk5" else n + 1), case["nelmt"]
    if case["kind"] == "bk1":
        geometry = 0.5 + torch.rand(e * nq ** 3, dtype=torch.float64, device="cuda", generator=g)
    else:
        geometry = 0.2 * torch.rand((e, 6, nq ** 3), dtype=torch.float64, device="cuda", generator=g)
        geometry[:, (0, 3, 5)] += 1.0
        geometry = geometry.view(-1)
    x = _gll(n)[0]
    xq = x if case["kind"] == "bk5" else np.polynomial.legendre.leggauss(nq)[0]
    def on(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return dict(B=on(_lagrange(x, xq)[0]), D=on(_lagrange(xq, xq)[1]), geometry=geometry, u=_uniform(e * n ** 3, g))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("bk1", "bk3", "bk5"):
        s = _element_inputs(case, seed)
        return dict(s, case=case, out=torch.empty_like(s["u"]))
    if kind == "batch":
        meshes, _ = mf.batch_workload(case["problems"], seed=case["mix"], cells=(6, 24))
        solver = mf.BatchSolver(meshes)
        g = np.random.default_rng(seed)
        b = solver.rhs_uniform(g.integers(0, 2 ** 63, case["problems"]))
        return dict(case=case, solver=solver, b=b, x=solver.initialize_dof_vector())
    mesh = _mesh(case)
    op = mf.LaplaceOperator(mesh, arith=case["arith"], quadrature=case["form"])
    src = _uniform(op.m() * (3 if kind == "vector" else 1), _generator(seed))
    s = dict(case=case, op=op, src=src, dst=torch.zeros_like(src))
    if kind == "host":
        s["src"] = src.cpu().pin_memory()
        s["dst"] = torch.zeros_like(s["src"]).pin_memory()
    elif kind in ("cg", "mg"):
        s["src"] = _interior(case, src)
        s["control"] = mf.ReductionControl(100000, 1e-300, case["reduce"])
        s["preconditioner"] = (op.get_matrix_diagonal_inverse() if kind == "cg"
                               else mf.MGPreconditioner(mesh, precision=32, operator=op))
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        return state["op"].vmult(state["dst"], state["src"])
    if kind == "vector":
        return state["op"].vmult_vector(state["dst"], state["src"])
    if kind == "host":
        return state["op"].vmult_host(state["dst"], state["src"])
    if kind == "bk1":
        return mf.bk1_evector(case["p"], state["B"], state["geometry"], state["u"], state["out"], arith=case["arith"])
    if kind == "bk3":
        return mf.bk3_evector(case["p"], state["B"], state["D"], state["geometry"], state["u"], state["out"],
                              arith=case["arith"])
    if kind == "bk5":
        return mf.bk5_evector(case["p"], state["D"], state["geometry"], state["u"], state["out"], arith=case["arith"])
    if kind == "batch":
        return state["solver"].solve(state["x"].zero_(), state["b"], max_steps=200, reduce=case["reduce"])
    x = state["dst"].zero_()
    return mf.SolverCG(state["control"]).solve(state["op"], x, state["src"], state["preconditioner"])


# ---- what a pass cannot do without -----------------------------------------
def _apply_work(cells, dofs, n, nq, components=1, word=8, mass=False):
    """Vectors once each way, the dof map, 6 (7) geometric factors per point; the dense 1D contractions."""
    contract = 0 if nq == n else 4 * (nq * n ** 3 + nq ** 2 * n ** 2 + nq ** 3 * n)
    contract += 12 * nq ** 4 + (17 if mass else 15) * nq ** 3
    return (2 * word * components * dofs + cells * (4 * n ** 3 + (7 if mass else 6) * word * nq ** 3),
            components * cells * contract)


def _box_work(case, **more):
    p = case["p"]
    form = case["form"]
    cells = case["nx"] * case["ny"] * case["nz"]
    dofs = (p * case["nx"] + 1) * (p * case["ny"] + 1) * (p * case["nz"] + 1)
    nq = p + 2 if form == "bp3" else p + 1
    b, f = _apply_work(cells, dofs, p + 1, nq, mass=form == "helmholtz", **more)
    if form in ("gauss", "helmholtz"):  # interpolation to as many points as nodes
        f += cells * 12 * (p + 1) ** 4
    return b, f, dofs


def _mg_work(b, b32, f, dofs, iterations):
    """A Krylov step (operator, 8 vectors) and the finest level's 11 single-precision applications and 22 vectors."""
    return iterations * (b + 64 * dofs + 11 * b32 + 88 * dofs), iterations * 12 * f


def work(case):
    kind = case["kind"]
    if kind in ("bk1", "bk3", "bk5"):
        n, e = case["p"] + 1, case["nelmt"]
        nq = n if kind == "bk5" else n + 1
        factors = 1 if kind == "bk1" else 6
        flops = 0 if nq == n else 4 * (nq * n ** 3 + nq ** 2 * n ** 2 + nq ** 3 * n)
        flops += nq ** 3 if kind == "bk1" else 12 * nq ** 4 + 15 * nq ** 3
        return dict(bytes=e * 8 * (2 * n ** 3 + factors * nq ** 3), flops=e * flops)
    if kind == "batch":
        meshes, _ = mf.batch_workload(case["problems"], seed=case["mix"], cells=(6, 24))
        total = [0, 0]
        for m in meshes:
            box = dict(form="gll", p=m.degree, nx=m.nx, ny=m.ny, nz=m.nz)
            b, f, dofs = _box_work(box)
            for i, v in enumerate(_mg_work(b, _box_work(box, word=4)[0], f, dofs, 9)):
                total[i] += v
        return dict(bytes=total[0], flops=total[1])
    b, f, dofs = _box_work(case, components=3 if kind == "vector" else 1)
    if kind == "cg":  # the iterations of a Jacobi-preconditioned solve on this mesh, about
        steps = round((4.5 + 0.45 * case["p"]) * dofs ** (1 / 3) * -math.log10(case["reduce"]) / 10)
        return dict(bytes=steps * (b + 10 * 8 * dofs), flops=steps * (f + 10 * dofs))
    if kind == "mg":
        b, f = _mg_work(b, _box_work(case, word=4)[0], f, dofs, 11)
    return dict(bytes=b, flops=f)


# ---- the same results in 64 bits with plain torch ---------------------------
def _lagrange(nodes, points):
    """(values, derivatives) [point, node] of the Lagrange polynomials on `nodes`."""
    n = len(nodes)
    V, D = np.ones((len(points), n)), np.zeros((len(points), n))
    for b in range(n):
        others = [m for m in range(n) if m != b]
        for m in others:
            V[:, b] *= (points - nodes[m]) / (nodes[b] - nodes[m])
        for skip in others:
            t = np.full(len(points), 1 / (nodes[b] - nodes[skip]))
            for m in others:
                if m != skip:
                    t = t * (points - nodes[m]) / (nodes[b] - nodes[m])
            D[:, b] += t
    return V, D


def _gll(n):
    """Gauss-Lobatto-Legendre points and weights on [-1, 1]."""
    L = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate([[-1.0], np.sort(L.deriv().roots().real), [1.0]]) if n > 2 else np.array([-1.0, 1.0])
    for _ in range(3):  # Newton steps on the interior points
        d1, d2 = L.deriv(), L.deriv(2)
        if n > 2:
            x[1:-1] -= d1(x[1:-1]) / d2(x[1:-1])
    x = 0.5 * (x - x[::-1])
    return x, 2 / (n * (n - 1) * L(x) ** 2)


def _along(A, u, axis):
    """A [q, m] applied to axis -3, -2 or -1 of u."""
    return torch.movedim(torch.matmul(torch.movedim(u, axis, -1), A.T), -1, axis)


class _Box:
    """The box operator on one slab of cell layers at a time; u[z, y, x] with x fastest."""

    def __init__(self, case, keep=False):
        self.case, p, form = case, case["p"], case["form"]
        self.p, self.n = p, p + 1
        x, w = _gll(p + 1)
        if form == "gll":
            xq, wq = x, w
        else:
            xq, wq = np.polynomial.legendre.leggauss(p + (2 if form == "bp3" else 1))
        def on(a):
            return torch.from_numpy(np.ascontiguousarray(a)).cuda()
        self.x, self.w = on(x), on(wq)
        self.B, self.DB = (on(a) for a in _lagrange(x, xq))  # nodes -> points: values, derivatives
        self.D = on(_lagrange(xq, xq)[1])                    # at the points
        self.cells = case["nz"], case["ny"], case["nx"]
        self.dofs = [p * c + 1 for c in self.cells]
        layer = self.cells[1] * self.cells[2] * len(xq) ** 3
        self.layers = max(1, 30_000_000 // layer)
        self.kept = {} if keep else None

    def slabs(self):
        for z in range(0, self.cells[0], self.layers):
            yield z, min(self.cells[0], z + self.layers)

    def factors(self, z0, z1):
        """(G [6, cells, points], JxW) of a slab's cells."""
        if self.kept is not None and z0 in self.kept:
            return self.kept[z0]
        spans = [torch.arange(a, b, dtype=torch.float64, device="cuda") for a, b in
                 ((z0, z1), (0, self.cells[1]), (0, self.cells[2]))]
        node = [(s[:, None] + 0.5 * (self.x + 1)) / c for s, c in zip(spans, self.cells)]  # [cell, node]
        zz, yy, xx = (node[0][:, None, None, :, None, None], node[1][None, :, None, None, :, None],
                      node[2][None, None, :, None, None, :])
        s = 0.05 * torch.sin(2 * math.pi * xx) * torch.sin(2 * math.pi * yy) * torch.sin(2 * math.pi * zz)
        J = []  # J[d][a]: derivative of coordinate d (z, y, x) along reference axis a
        for coordinate in (zz, yy, xx):
            X = (coordinate + s).reshape(-1, self.n, self.n, self.n)
            row = []
            for a in (-3, -2, -1):
                t = X
                for b in (-3, -2, -1):
                    t = _along(self.DB if a == b else self.B, t, b)
                row.append(t)
            J.append(row)
        C = [[J[(d + 1) % 3][(a + 1) % 3] * J[(d + 2) % 3][(a + 2) % 3] -
              J[(d + 1) % 3][(a + 2) % 3] * J[(d + 2) % 3][(a + 1) % 3] for a in range(3)] for d in range(3)]
        det = sum(J[d][0] * C[d][0] for d in range(3))
        w = self.w[:, None, None] * self.w[:, None] * self.w
        G = [sum(C[d][a] * C[d][b] for d in range(3)) * (w / det) for a, b in
             ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
        r = G, det * w
        if self.kept is not None:
            self.kept[z0] = r
        return r

    def elements(self, u, z0, z1):
        """Element operators on u[cell, n, n, n]."""
        form = self.case["form"]
        G, JxW = self.factors(z0, z1)
        if form != "gll":
            for a in (-3, -2, -1):
                u = _along(self.B, u, a)
        q = [_along(self.D, u, a) for a in (-3, -2, -1)]
        v = [G[0] * q[0] + G[1] * q[1] + G[2] * q[2], G[1] * q[0] + G[3] * q[1] + G[4] * q[2],
             G[2] * q[0] + G[4] * q[1] + G[5] * q[2]]
        y = sum(_along(self.D.T, t, a) for t, a in zip(v, (-3, -2, -1)))
        if form == "helmholtz":
            y = y + JxW * u
        if form != "gll":
            for a in (-3, -2, -1):
                y = _along(self.B.T, y, a)
        return y

    def apply(self, src):
        """A src with identity rows on the boundary."""
        p, n = self.p, self.n
        full = src.view(self.dofs)
        inner = torch.zeros_like(full)
        inner[1:-1, 1:-1, 1:-1] = full[1:-1, 1:-1, 1:-1]
        out = torch.zeros_like(full)
        for z0, z1 in self.slabs():
            u = inner[p * z0:p * z1 + 1].unfold(0, n, p).unfold(1, n, p).unfold(2, n, p).contiguous()
            y = self.elements(u.view(-1, n, n, n), z0, z1).view(u.shape)
            for axis in (2, 1, 0):  # sum the cells' shares along x, then y, then z
                shape = list(y.shape[:-1])
                shape[axis] = p * (y.shape[axis]) + 1
                t = torch.zeros(shape, dtype=y.dtype, device=y.device)
                for k in range(n):
                    at = [slice(None)] * t.dim()
                    at[axis] = slice(k, k + p * (y.shape[axis] - 1) + 1, p)
                    t[tuple(at)] += y[..., k]
                y = t
            out[p * z0:p * z1 + 1] += y
        edge = torch.ones(self.dofs, dtype=torch.bool, device="cuda")
        edge[1:-1, 1:-1, 1:-1] = False
        out[edge] = full[edge]
        return out.view(-1)

    def diagonal(self):
        """Cheap approximation of the diagonal, enough to precondition: the point terms of G."""
        d = torch.zeros(self.dofs, dtype=torch.float64, device="cuda")
        D2 = self.D.square()
        n, p = self.n, self.p
        for z0, z1 in self.slabs():
            G, _ = self.factors(z0, z1)
            y = sum(_along(D2.T, G[c], a) for c, a in ((0, -3), (3, -2), (5, -1)))
            y = y.view(z1 - z0, self.cells[1], self.cells[2], n, n, n)
            for k in np.ndindex(n, n, n):
                at = tuple(slice(s + k_, s + k_ + p * (c - 1) + 1, p) for s, k_, c in
                           zip((p * z0, 0, 0), k, y.shape[:3]))
                d[at] += y[(...,) + k]
        return d.view(-1)


def _solve(box, b, reduce, most=20000):
    inverse = 1 / box.diagonal()
    x, r = torch.zeros_like(b), b.clone()
    z = inverse * r
    q, rz, goal = z.clone(), torch.dot(r, z), reduce * float(b.norm())
    for k in range(most):
        v = box.apply(q)
        a = rz / torch.dot(q, v)
        x += a * q
        r -= a * v
        if k % 10 == 0 and float(r.norm()) <= goal:
            return x
        z = inverse * r
        new = torch.dot(r, z)
        q = z + (new / rz) * q
        rz = new
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bk1", "bk3", "bk5"):
        s, n = _element_inputs(case, seed), case["p"] + 1
        B, D, u = s["B"], s["D"], s["u"].view(-1, n, n, n)
        axes = (-3, -2, -1)
        if kind != "bk5":
            for a in axes:
                u = _along(B, u, a)
        if kind == "bk1":
            u = u * s["geometry"].view(u.shape)
        else:
            G = s["geometry"].view(case["nelmt"], 6, *u.shape[1:])
            q = [_along(D, u, a) for a in axes]
            v = [sum(G[:, c] * t for c, t in zip(row, q)) for row in ((0, 1, 2), (1, 3, 4), (2, 4, 5))]
            u = sum(_along(D.T, t, a) for t, a in zip(v, axes))
        if kind != "bk5":
            for a in axes:
                u = _along(B.T, u, a)
        return u.reshape(-1)
    if kind == "batch":
        return None  # a solve for each problem: too long
    components = 3 if kind == "vector" else 1
    solve = kind in ("cg", "mg")
    dofs = math.prod(case["p"] * case[d] + 1 for d in ("nx", "ny", "nz"))
    if solve and dofs > SOLVE_LIMIT:
        return None
    box = _Box(case, keep=solve)
    src = _uniform(dofs * components, _generator(seed))
    if solve:
        return _solve(box, _interior(case, src), 1e-13)
    out = torch.stack([box.apply(src[c::components].contiguous()) for c in range(components)], -1).view(-1)
    return out.cpu() if kind == "host" else out
