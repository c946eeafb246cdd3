"""Multigrid CG on operators built from a caller's arrays, whose identity rows are
not the hierarchy's masked ones: a map that leaves the constrained DoFs in, more
constrained DoFs than the box boundary, fewer of them.

Tolerances, before the first run: the solves stop at a recursive residual of 1e-12,
so the true one is within 1e-10 of |b| (the gap between the two stays near rounding
times the condition number, at most about 1e4 on these meshes) and the solution
within 1e-7 of Jacobi-CG's (condition number times both residuals)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def full_map(cells, p):
    """[cell][(p + 1)^3] DoF of every local node, none masked (x fastest)."""
    nx, ny, nz = cells
    X, Y = p * nx + 1, p * ny + 1
    k, j, i = np.meshgrid(*(np.arange(p + 1),) * 3, indexing="ij")
    cz, cy, cx = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    node = (i + X * (j + Y * k)).reshape(1, -1)
    return (p * (cx + X * (cy + Y * cz)).reshape(-1, 1) + node).astype(np.uint32).reshape(-1)


@pytest.mark.parametrize("p,cells", [(1, (6, 5, 8)), (3, (5, 4, 4))])
@pytest.mark.parametrize("kind", ["unmasked", "more", "fewer"])
@pytest.mark.parametrize("precision", [32, 64])
def test_mg_cg_takes_the_operators_own_identity_rows(orc, p, cells, kind, precision):
    import torch

    import benchmarks_gb300 as mf
    ref = orc.BoxProblem(*cells, p, amplitude=0.05)
    n = ref.n_dofs
    whole = full_map(cells, p)
    valid = ref.map != 0xFFFFFFFF
    assert np.array_equal(whole[valid], ref.map[valid])
    boundary = np.asarray(ref.constrained, dtype=np.int64)
    rng = np.random.default_rng(p)
    b = rng.uniform(-1, 1, n)
    if kind == "unmasked":
        # (rows of the boundary are 0 in b: the operator is symmetric only there)
        constrained, dof_map = boundary, whole
        b[boundary] = 0.0
    else:
        if kind == "more":
            inner = np.setdiff1d(np.arange(n), boundary)
            constrained = np.sort(np.concatenate([boundary, rng.choice(inner, inner.size // 10, replace=False)]))
        else:  # one face
            constrained = np.arange((p * cells[0] + 1) * (p * cells[1] + 1), dtype=np.int64)
        dof_map = np.where(np.isin(whole, constrained), np.uint32(0xFFFFFFFF), whole)
    A = mf.LaplaceOperator(degree=p, n_dofs=n, dof_map=dof_map, G=ref.G, constrained=constrained)
    M = mf.MGPreconditioner(mf.BoxMesh(*cells, degree=p, amplitude=0.05), precision=precision)
    bt = torch.from_numpy(b).cuda()
    control = mf.ReductionControl(3000, 1e-300, 1e-12)
    x, y = A.initialize_dof_vector(), A.initialize_dof_vector()
    mf.SolverCG(control).solve(A, x, bt, M)
    A.vmult(y, x)
    assert rel(y.cpu().numpy(), b) <= 1e-10
    want = A.initialize_dof_vector()
    mf.SolverCG(control).solve(A, want, bt, A.get_matrix_diagonal_inverse())
    assert rel(x.cpu().numpy(), want.cpu().numpy()) <= 1e-7
