"""Values on Dirichlet rows do not reach the interior rows of a V-cycle whose finest
level is Q1: infinities, NaN and values beyond FP32 there are masked, as the
operators mask them.

Tolerance, before the first run: the interior rows equal those of the same vector
with zeros on the boundary to 1e-6 relative, the rounding of the FP32 V-cycle (the
masked values enter no sum; atomics may reorder the others)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def interior(cells, p):
    n = [p * c + 1 for c in reversed(cells)]
    m = np.zeros(n, dtype=bool)
    m[1:-1, 1:-1, 1:-1] = True
    return m.reshape(-1)


# (extents that halve evenly: a narrower last cell restricts the boundary row's residual too)
@pytest.mark.parametrize("cells,cheb", [((8, 8, 8), 3), ((16, 8, 32), 2), ((8, 8, 8), 1)])
@pytest.mark.parametrize("value", [np.inf, np.nan, 1e300])
def test_boundary_values_stay_on_the_boundary(cells, cheb, value):
    import torch

    import benchmarks_gb300 as mf
    mesh = mf.BoxMesh(*cells, degree=1, amplitude=0.05)
    M = mf.MGPreconditioner(mesh, precision=32, chebyshev_degree=cheb, coarse_cells=4)
    B = mf.BatchSolver([mesh, mf.BoxMesh(4, 4, 4, degree=2)], chebyshev_degree=cheb, coarse_cells=4)
    inside = interior(cells, 1)
    r = np.random.default_rng(2).uniform(-1, 1, mesh.n_dofs)
    r[~inside] = 0.0
    z = []
    for v in (0.0, value):
        r[~inside] = v
        rt = torch.from_numpy(r).cuda()
        zt = torch.empty_like(rt)
        M.vmult(zt, rt)
        rb = torch.zeros(B.n_dofs, dtype=torch.float64, device="cuda")
        zb = torch.empty_like(rb)
        B.split(rb)[0].copy_(rt)
        B.precondition(zb, rb)
        z.append((zt.cpu().numpy()[inside], B.split(zb)[0].cpu().numpy()[inside]))
    for clean, got in zip(*z):
        assert np.isfinite(got).all()
        assert np.linalg.norm(got - clean) <= 1e-6 * np.linalg.norm(clean)
