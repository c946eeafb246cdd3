"""Q1 multigrid levels smoothed by assembled stencils (FP32 V-cycle).

Tolerances, before the first run: the FP32 V-cycle against the FP64 oracle 1e-4
relative, the batched one against the single-problem one 1e-5 relative (the
bounds of the other V-cycle tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# boxes of one interior node a direction, of less than a block, over block edges, of odd counts and
# unlike extents; smoothers of degree 1 (by the operator), of one and of several stencil steps
# (every smoothed level has an interior node, without one lambda_max is 0 / 0 in the oracle)
@pytest.mark.parametrize("box,cheb,coarse", [
    ((2, 3, 2), 2, 2), ((5, 3, 9), 1, 4), ((5, 3, 9), 2, 4), ((8, 7, 11), 3, 2), ((33, 6, 4), 4, 17),
    ((16, 17, 15), 5, 2)])
@pytest.mark.parametrize("p", [1, 2])
def test_vcycle_over_q1_levels(box, cheb, coarse, p):
    import benchmarks_gb300 as mf
    from oracle import mg_oracle
    mesh = mf.BoxMesh(*box, degree=p, amplitude=0.08)
    M = mf.MGPreconditioner(mesh, precision=32, coarse_cells=coarse, chebyshev_degree=cheb)
    A = mf.LaplaceOperator(mesh)
    r, z = A.rhs_uniform(3), A.initialize_dof_vector()
    M.vmult(z, r)
    mgo = mg_oracle.MGOracle(*box, p, amplitude=0.08, coarse_cells=coarse, chebyshev_degree=cheb)
    assert rel(z.cpu().numpy(), mgo.vcycle(r.cpu().numpy())) <= 1e-4
    B = mf.BatchSolver([mesh, mf.BoxMesh(4, 4, 4, degree=3), mesh], coarse_cells=coarse,
                       chebyshev_degree=cheb)
    rb, zb = B.rhs_uniform([3, 4, 5]), B.initialize_dof_vector()
    B.precondition(zb, rb)
    assert rel(B.split(zb)[0].cpu().numpy(), z.cpu().numpy()) <= 1e-5
    M.vmult(z, B.split(rb)[2].contiguous())
    assert rel(B.split(zb)[2].cpu().numpy(), z.cpu().numpy()) <= 1e-5
