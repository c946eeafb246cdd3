"""Q1 stencils and device memory: a hierarchy and a batch take them whatever else holds
memory, end in less memory than with the operators' FP32 factors, and fall back to the
operators where an allocation for them fails; nothing that fitted without them fails.

Tolerance, before the first run: V-cycles with and without stencils agree to 1e-5 relative
(the bound between FP32 V-cycles of the other tests)."""
import ctypes
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stencils(M=None, B=None):
    import benchmarks_gb300 as mf
    from benchmarks_gb300 import _abi
    n = ctypes.c_int(-1)
    _abi.check(mf.lib().mfgb_test_stencil_levels(M._mg if M else None, B._b if B else None, ctypes.byref(n)))
    return n.value


def free():
    import torch
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_stencils_do_not_depend_on_free_memory():
    import torch

    import benchmarks_gb300 as mf
    mesh = mf.BoxMesh(128, 128, 128, degree=1)
    levels = stencils(mf.MGPreconditioner(mesh, precision=32))
    assert levels == 5
    # the set-up's own need (about 1.6 GB) and little more stay free
    hold = torch.empty(free() - (1750 << 20), dtype=torch.uint8, device="cuda")
    assert stencils(mf.MGPreconditioner(mesh, precision=32)) == levels
    del hold


def test_hierarchy_ends_in_no_more_memory_than_with_operators():
    import benchmarks_gb300 as mf
    mesh = mf.BoxMesh(96, 96, 96, degree=1)
    used = {}
    for cheb in (1, 3):  # smoothed by operators, by stencils
        before = free()
        M = mf.MGPreconditioner(mesh, precision=32, chebyshev_degree=cheb)
        used[stencils(M) > 0] = before - free()
        del M
    assert used[True] <= used[False]


@pytest.mark.parametrize("what", ["hierarchy", "shared", "batch"])
def test_failed_stencil_allocation_smooths_by_operators(what):
    import torch

    import benchmarks_gb300 as mf
    from benchmarks_gb300 import MfgbError, _abi
    L = mf.lib()
    mesh = mf.BoxMesh(12, 9, 10, degree=1, amplitude=0.05)
    A = mf.LaplaceOperator(mesh)
    r = A.rhs_uniform(1)

    def build():
        if what == "batch":
            S = mf.BatchSolver([mesh, mf.BoxMesh(6, 6, 6, degree=2)])
            rb = torch.zeros(S.n_dofs, dtype=torch.float64, device="cuda")
            S.split(rb)[0].copy_(r)
            z = torch.empty_like(rb)
            S.precondition(z, rb)
            return stencils(B=S), S.split(z)[0].cpu().numpy()
        M = mf.MGPreconditioner(mesh, precision=32, operator=A if what == "shared" else None)
        z = torch.empty_like(r)
        M.vmult(z, r)
        return stencils(M), z.cpu().numpy()

    most, want = build()
    assert most >= 1
    seen, done = set(), 0
    try:
        for n in range(1, 400):
            before = free()
            _abi.check(L.mfgb_test_fail_allocation(n))
            try:
                levels, z = build()
                seen.add(levels)
                assert np.linalg.norm(z - want) <= 1e-5 * np.linalg.norm(want)
                done = done + 1 if levels == most else 0
            except MfgbError as e:
                assert e.status == _abi.ERR_OUT_OF_MEMORY
                done = 0
            finally:
                _abi.check(L.mfgb_test_fail_allocation(0))
            assert free() >= before - (2 << 20)
            if done == 3:  # past the last allocation
                break
    finally:
        _abi.check(L.mfgb_test_fail_allocation(0))
    assert done == 3
    assert min(seen) < most  # some set-up went on without a stencil


def test_smoother_weights_and_solve_on_a_level_without_factors():
    """The factors a stencil replaced come back for the lambda_max estimate of new weights."""
    import torch

    import benchmarks_gb300 as mf
    from benchmarks_gb300 import _abi
    mesh = mf.BoxMesh(10, 8, 9, degree=1, amplitude=0.05)
    A = mf.LaplaceOperator(mesh)
    M = mf.MGPreconditioner(mesh, precision=32)
    r, z0, z1 = A.rhs_uniform(2), A.initialize_dof_vector(), A.initialize_dof_vector()
    M.vmult(z0, r)
    w = torch.ones(mesh.n_cells, dtype=torch.float64, device="cuda")
    _abi.check(mf.lib().mfgb_mg_set_smoother_weights(M._mg, ctypes.c_void_p(w.data_ptr())))
    M.vmult(z1, r)  # unit weights: the plain diagonal again
    assert float(torch.linalg.norm(z1 - z0) / torch.linalg.norm(z0)) <= 1e-5
    x = A.initialize_dof_vector()
    control = mf.ReductionControl(100, 1e-300, 1e-10)
    mf.SolverCG(control).solve(A, x, r, M)
    assert control.last_step() <= 25
