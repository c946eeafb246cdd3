"""Which FP64 GLL kernel an application takes: the line kernel for an operator's own
arrays from degree 5, and for everything it does not cover (element vectors, arrays
off 16 bytes, matrices without the mirror symmetry) the kernel that is fastest there,
which at degrees 6 and 8 is point-per-thread and not the column kernel."""
import ctypes

import numpy as np
import pytest

COLUMN, POINT, TMA, COLUMN_ALT, TMA_ALT, LINE = 0, 1, 2, 3, 4, 7


def shape(degree, evector, aligned, mirror):
    import benchmarks_gb300 as mf
    from benchmarks_gb300 import _abi
    out = ctypes.c_int(-1)
    _abi.check(mf.lib().mfgb_test_fp64_shape(degree, evector, aligned, mirror, ctypes.byref(out)))
    return out.value


@pytest.mark.parametrize("degree,evector,general,unaligned,own", [
    (1, COLUMN, TMA_ALT, COLUMN, TMA_ALT), (2, COLUMN, COLUMN_ALT, COLUMN_ALT, COLUMN_ALT),
    (3, COLUMN, TMA, COLUMN, TMA), (4, COLUMN, TMA_ALT, COLUMN, TMA_ALT), (5, COLUMN, TMA, COLUMN, LINE),
    (6, POINT, POINT, POINT, LINE), (7, COLUMN, TMA, COLUMN, LINE), (8, POINT, POINT, POINT, LINE)])
def test_shape_of_every_kind_of_call(degree, evector, general, unaligned, own):
    for aligned in (0, 1):
        for mirror in (0, 1):
            assert shape(degree, 1, aligned, mirror) == evector
    assert shape(degree, 0, 1, 0) == general
    assert shape(degree, 0, 0, 0) == shape(degree, 0, 0, 1) == unaligned
    assert shape(degree, 0, 1, 1) == own


@pytest.mark.gpu
@pytest.mark.parametrize("p", [5, 6, 7, 8])
@pytest.mark.parametrize("offset", [0, 1])  # doubles the arrays start past 16 bytes
def test_seams_match_oracle(p, offset):
    """Cell counts around the cells per thread block; tolerance of the FP64 arithmetic, 1e-13."""
    import torch

    import benchmarks_gb300 as mf
    from oracle import oracle
    n = p + 1
    rng = np.random.default_rng(p)
    general = rng.uniform(-1, 1, (n, n))

    def on(a):
        t = torch.empty(a.size + offset, dtype=torch.float64, device="cuda")[offset:]
        return t.copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1)))
    for D in (general, 0.5 * (general - general[::-1, ::-1])):
        for cells in (1, 2, 11):
            G = rng.uniform(-1, 1, cells * 6 * n ** 3)
            u = rng.uniform(-1, 1, cells * n ** 3)
            want = oracle.evector(n, D, G, u)
            Dt, Gt, ut = on(D), on(G), on(u)
            got = mf.bk5_evector(p, Dt, Gt, ut, torch.zeros_like(ut), arith="fp64").cpu().numpy()
            assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)
            index = torch.arange(cells * n ** 3, dtype=torch.int32, device="cuda")
            got = mf.bk5_lvector(p, Dt, Gt, ut, torch.zeros_like(ut), index, arith="fp64").cpu().numpy()
            assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)
