"""The line contractions of the double-float kernels (benchmarks_gb300/csrc/
mfgb_fxline.cuh: fx_grid, fx_line, fx_sum3 in even-odd form) restated with numpy
float32 operations.

Claims checked: rounding a line to the grid of 3 max|x| leaves the sums and
differences of mirrored values exact; with the offset max(bound A, bound B) + bound(A +- B)
the high parts of A +- B add exactly; the result is as accurate as the plain offset sum
(2^-42 of the bound at most, near 2^-46 in the mean); and on the GPU a caller's
general derivative matrix takes the plain form, a mirror-antisymmetric one the
even-odd form, both to 1e-12 of the oracle."""
import numpy as np
import pytest

from test_fx_arith import Acc, EXT, ext, f32, gll_derivative, split

extended = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 60, reason="needs an extended long double")


def grid(x, C):
    t = (C + x[0]).astype(f32)
    h = (t - C).astype(f32)
    return h, ((x[0] - h).astype(f32) + x[1]).astype(f32)


def add(a, b, sign=1):
    """(sum of the parts, whether the high parts' sum is exact)"""
    h = (a[0] + f32(sign) * b[0]).astype(f32)
    exact = np.all(h.astype(EXT) == a[0].astype(EXT) + sign * b[0].astype(EXT))
    return (h, (a[1] + f32(sign) * b[1]).astype(f32)), bool(exact)


def line(M, x, sym):
    """fx_line for mirror-symmetric (sym = 1) or antisymmetric (-1) M; x: pairs per input"""
    no, ni = M.shape
    hi, ok = ni // 2, True
    mx = (np.max([np.abs(v[0]) for v in x], axis=0) * f32(1 + 2.0 ** -20)).astype(f32)
    C = (mx * f32(3)).astype(f32)
    x = [v if ni % 2 and i == hi else grid(v, C) for i, v in enumerate(x)]
    e, f = [], []
    for i in range(hi):
        s, k1 = add(x[i], x[ni - 1 - i])
        d, k2 = add(x[i], x[ni - 1 - i], -1)
        e.append(s), f.append(d)
        ok &= k1 and k2
    y, bound = [None] * no, []
    for o in range((no + 1) // 2):
        P = [split(0.5 * (M[o, i] + M[o, ni - 1 - i])) for i in range(hi)]
        Q = [split(0.5 * (M[o, i] - M[o, ni - 1 - i])) for i in range(hi)]
        xs = list(e)
        if ni % 2:
            P.append(split(M[o, hi])), xs.append(x[hi])
        bp = sum((2 if i < hi else 1) * abs(float(p[0])) for i, p in enumerate(P))
        bq = sum(2 * abs(float(q[0])) for q in Q)
        row = sum(2 * max(abs(float(p[0])), abs(float(q[0]))) for p, q in zip(P, Q)) + \
            (abs(float(P[hi][0])) if ni % 2 else 0)
        Co = (f32((1 + 2.0 ** -18) * (max(bp, bq) + row)) * mx).astype(f32)
        bound.append(Co)
        A, B = Acc(Co), Acc(Co)
        for p, v in zip(P, xs):
            A.add((np.full_like(mx, p[0]), np.full_like(mx, p[1])), v)
        for q, v in zip(Q, f):
            B.add((np.full_like(mx, q[0]), np.full_like(mx, q[1])), v)
        a, b = A.finish(), B.finish()
        ok &= A.exact_ok and B.exact_ok
        if no % 2 and o == no // 2:
            y[o] = b if sym < 0 else a
        else:
            y[o], k1 = add(a, b)
            y[no - 1 - o], k2 = add(b, a, -1) if sym < 0 else add(a, b, -1)
            ok &= k1 and k2
    return y, np.max(bound, axis=0), ok


@extended
@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("spread", [0, 12])  # binades between a line's values
def test_line_in_even_odd_form(n, spread):
    D = gll_derivative(n)[1]
    D = 0.5 * (D - D[::-1, ::-1])
    rng = np.random.default_rng(n)
    x = [split(rng.uniform(-1, 1, 3000) * 2.0 ** -rng.integers(0, spread + 1, 3000)) for _ in range(n)]
    for M in (D, D.T.copy()):
        y, C, ok = line(M, x, -1)
        assert ok
        Mp = [[split(M[o, i]) for i in range(n)] for o in range(n)]
        err = np.array([np.abs(ext(y[o]) - sum(ext(Mp[o][i]) * ext(x[i]) for i in range(n))) / C.astype(EXT)
                        for o in range(n)])
        assert float(err.max()) < 2.0 ** -42
        assert float(np.sqrt(np.mean(err ** 2))) < 2.0 ** -45


@extended
def test_sum_of_three_shares():
    rng = np.random.default_rng(3)
    v = [split(rng.uniform(-1, 1, 20000) * 2.0 ** rng.integers(-20, 20, 20000)) for _ in range(3)]
    (a, al), (b, bl), (c, cl) = v
    s = a + b
    bb = s - a
    e = (a - (s - bb)) + (b - bb)
    t = s + c
    cc = t - s
    g = (s - (t - cc)) + (c - cc)
    lo = ((al + bl) + (e + g)) + cl
    big = np.max([np.abs(x[0]) for x in v], axis=0).astype(EXT)
    assert float(np.max(np.abs(ext((t, lo)) - sum(map(ext, v))) / big)) < 2.0 ** -45


@pytest.mark.gpu
@pytest.mark.parametrize("p", range(1, 9))
def test_seam_matrices_of_both_kinds(p):
    """Cell counts around the cells per thread block and the dof-map windows' ends."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import benchmarks_gb300 as mf
    from oracle import oracle
    n = p + 1
    rng = np.random.default_rng(p)
    general = rng.uniform(-1, 1, (n, n))
    for D in (general, 0.5 * (general - general[::-1, ::-1])):
        for cells in (1, 2, 7, 37):
            G = rng.uniform(-1, 1, cells * 6 * n ** 3)
            u = rng.uniform(-1, 1, cells * n ** 3)
            want = oracle.evector(n, D, G, u)
            dev = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (D, G, u)]
            got = mf.bk5_evector(p, *dev, torch.zeros_like(dev[2]), arith="df").cpu().numpy()
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
            index = torch.arange(cells * n ** 3, dtype=torch.int32, device="cuda")
            got = mf.bk5_lvector(p, *dev, torch.zeros_like(dev[2]), index, arith="df").cpu().numpy()
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("p", range(1, 9))
def test_interpolation_seams_of_both_kinds(p):
    """BK1 and BK3 with mirror-symmetric and general matrices, element counts around the cells per
    thread block."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import benchmarks_gb300 as mf
    from oracle import oracle
    n, q = p + 1, p + 2
    rng = np.random.default_rng(p)
    B, D = rng.uniform(-1, 1, (q, n)), rng.uniform(-1, 1, (q, q))
    for b, d in ((B, D), (0.5 * (B + B[::-1, ::-1]), 0.5 * (D - D[::-1, ::-1]))):
        for cells in (1, 5, 29):
            G, J = rng.uniform(-1, 1, cells * 6 * q ** 3), rng.uniform(0.5, 1.5, cells * q ** 3)
            u = rng.uniform(-1, 1, cells * n ** 3)
            db, dd, dG, dJ, du = (torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()
                                  for a in (b, d, G, J, u))
            got = mf.bk3_evector(p, db, dd, dG, du, torch.zeros_like(du), arith="df").cpu().numpy()
            want = oracle.bk3_evector(n, q, b, d, G, u)
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
            got = mf.bk1_evector(p, db, dJ, du, torch.zeros_like(du), arith="df").cpu().numpy()
            want = oracle.bk1_evector(n, q, b, J, u)
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("p", range(1, 9))
def test_plain_line_kernels(p):
    """FP32 (shapes 2 and 4) and FP64 operators on meshes of one cell, of odd cell counts that leave
    partial batches and unaligned tiles, and of several batches a thread block."""
    import ctypes

    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import benchmarks_gb300 as mf
    from benchmarks_gb300 import _abi
    from oracle import oracle
    L = mf.lib()
    old = {a: ctypes.c_int() for a in (0, 2)}
    for a in old:
        L.mfgb_get_kernel_shape(a, p, ctypes.byref(old[a]))
    big = {1: 60, 2: 44, 3: 34, 4: 30, 5: 26, 6: 22, 7: 20, 8: 18}[p]
    try:
        for cells in ((1, 1, 1), (3, 5, 3), (big, big - 1, big + 1)):
            A = mf.LaplaceOperator(mf.BoxMesh(*cells, degree=p))
            ref = oracle.BoxProblem(*cells, p, amplitude=0.05)
            src = np.random.default_rng(p).uniform(-1, 1, ref.n_dofs)
            want = ref.apply(src)
            u64 = torch.from_numpy(src).cuda()
            for shape in (2, 4):
                for a, dt, bound in ((0, torch.float64, 1e-12), (2, torch.float32, 1e-5)):
                    _abi.check(L.mfgb_set_kernel_shape(a, p, shape))
                    u = u64.to(dt)
                    y = torch.zeros_like(u)
                    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (y, u)]
                    _abi.check(L.mfgb_vmult_f32(A.handle, *ptr, None) if a == 2 else
                               L.mfgb_vmult(A.handle, *ptr, 0, None))
                    torch.cuda.synchronize()
                    mf.check_device_errors()
                    got = y.double().cpu().numpy()
                    assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want), (cells, shape, a)
    finally:
        for a, v in old.items():
            L.mfgb_set_kernel_shape(a, p, v.value)


@pytest.mark.gpu
def test_start_values_of_masked_and_unmasked_operators():
    """Identity rows and cleared rows before the cell loop: vector lengths around the 256 entries a
    warp clears, unaligned results, three components; a caller's map that leaves constrained DoFs
    in keeps their rows as plain copies."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import benchmarks_gb300 as mf
    from oracle import oracle
    rng = np.random.default_rng(0)
    for cells, p in (((1, 1, 1), 1), ((2, 1, 1), 4), ((6, 5, 7), 1), ((9, 11, 10), 2)):
        A = mf.LaplaceOperator(mf.BoxMesh(*cells, degree=p))
        ref = oracle.BoxProblem(*cells, p, amplitude=0.05)
        n = ref.n_dofs
        src = rng.uniform(-1, 1, n)
        want = ref.apply(src)
        for shift in (0, 1):
            u = torch.from_numpy(np.concatenate([np.zeros(shift), src])).cuda()[shift:]
            y = torch.full((n + shift,), 7.0, dtype=torch.float64, device="cuda")[shift:]
            for arith in ("df", "fp64"):
                got = A.vmult(y.fill_(7.0), u, arith=arith).cpu().numpy()
                assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
                assert np.array_equal(got[ref.constrained], src[ref.constrained])
        v = np.stack([src, 2 * src, -src], -1).reshape(-1)
        got = A.vmult_vector(torch.full((3 * n,), 7.0, dtype=torch.float64, device="cuda"),
                             torch.from_numpy(v).cuda()).cpu().numpy()
        w = np.stack([want, 2 * want, -want], -1).reshape(-1)
        assert np.linalg.norm(got - w) <= 1e-12 * np.linalg.norm(w)
    # constrained DoFs left in the map: their rows are overwritten by the source
    p, cells = 3, 4
    nn = (p + 1) ** 3
    dof_map = np.arange(cells * nn, dtype=np.uint32)
    fixed = np.array([0, 5, nn, 3 * nn + 7], dtype=np.int64)
    G = rng.uniform(0.5, 1.5, cells * 6 * nn)
    B = mf.LaplaceOperator(degree=p, n_dofs=cells * nn, dof_map=dof_map, G=G, constrained=fixed)
    D = oracle.derivative_matrix(oracle.gll(p + 1)[0])
    src = rng.uniform(-1, 1, cells * nn)
    want = oracle.apply(p + 1, dof_map, D, G, cells * nn, fixed, src)
    u = torch.from_numpy(src).cuda()
    got = B.vmult(torch.zeros_like(u), u).cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
    assert np.array_equal(got[fixed], src[fixed])


@pytest.mark.gpu
@pytest.mark.parametrize("quadrature,p,n", [("bp3", 5, 18), ("bp3", 5, 19), ("gauss", 6, 15), ("gauss", 6, 16)])
def test_start_values_beside_and_after_the_wide_kernels(quadrature, p, n):
    """Both sides of the 8e5 values above which a Gauss-point kernel of 7 points a direction begins
    after its start values, twice into a result that held something else.  1e-12 as for every apply."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import benchmarks_gb300 as mf
    from oracle import oracle
    A = mf.LaplaceOperator(mf.BoxMesh(n, n, n, degree=p, amplitude=0.05), quadrature=quadrature)
    ref = oracle.GaussProblem(n, n, n, p, nq=7, amplitude=0.05)
    assert (A.m() > 800000) == (n in (19, 16))
    src = np.random.default_rng(n).uniform(-1, 1, A.m())
    want = ref.apply(src)
    u, y = torch.from_numpy(src).cuda(), torch.full((A.m(),), 7.0, dtype=torch.float64, device="cuda")
    for _ in range(2):
        got = A.vmult(y, u).cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
