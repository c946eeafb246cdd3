"""Error of the double-float collocation kernel on values that are not spread evenly
(benchmarks_gb300/csrc/mfgb_bk5fx.cuh), against the plain form of its arithmetic: one
offset sum an output, pairs of 48 bits, restated with numpy float32 operations.

Tolerance, before the first run: the kernel's error (2-norm, against extended precision)
is no larger than the plain form's."""
import numpy as np
import pytest

from test_fx_arith import Acc, EXT, K, f32, gll_derivative, split

extended = pytest.mark.skipif(np.finfo(np.longdouble).nmant < 60, reason="needs an extended long double")
ROWS = ((0, 1, 2), (1, 3, 4), (2, 4, 5))


def along(u, axis, i):
    return tuple(np.take(v, [i], axis=axis + 1) for v in u)


def pair_of(value, like):
    h, l = split(value)
    return np.full_like(like, h), np.full_like(like, l)


def truncated(x):
    """fx_from_double: 24 bits, and the rest in 24"""
    m, e = np.frexp(x)
    h = np.ldexp(np.trunc(m * 2 ** 24), e - 24)
    return h.astype(f32), (x - h).astype(f32)


def plain(D, u, G):
    """(hi, lo) of the element operator on u [cell, n, n, n], |u| < 1, G six pairs of the same shape"""
    n = len(D)
    x, ones = truncated(u), np.ones_like(u, dtype=f32)
    rows = [K * f32(np.abs(D[i].astype(f32)).sum()) for i in range(n)]
    q = []
    for a in range(3):
        out = []
        for i in range(n):
            first = along(x, a, 0)[0]
            s = Acc(np.full_like(first, rows[i]))
            for m in range(n):
                s.add(pair_of(D[i, m], first), along(x, a, m))
            out.append(s.finish())
        q.append(tuple(np.concatenate([v[c] for v in out], axis=a + 1) for c in (0, 1)))
    kq = (K * np.max([np.abs(v[0]) for v in q], axis=0)).astype(f32)
    flux = []
    for r in ROWS:
        s = Acc((sum(np.abs(G[g][0]) for g in r) * kq).astype(f32))
        for g, v in zip(r, q):
            s.add(G[g], v)
        flux.append(s.finish())
    cols = [K * f32(np.abs(D[:, i].astype(f32)).sum()) for i in range(n)]
    C = 0
    for a in range(3):
        shape = [1, 1, 1, 1]
        shape[a + 1] = n
        C = C + np.max(np.abs(flux[a][0]), axis=a + 1, keepdims=True) * np.array(cols, f32).reshape(shape)
    s = Acc((C * ones).astype(f32))
    for m in range(n):
        for a in range(3):
            shape = [1, 1, 1, 1]
            shape[a + 1] = n
            d = [np.broadcast_to(v.reshape(shape), u.shape) for v in split(D[m])]
            s.add(d, [np.broadcast_to(v, u.shape) for v in along(flux[a], a, m)])
    return s.finish()


def exact(D, u, G):
    D, u, G = D.astype(EXT), u.astype(EXT), [g.astype(EXT) for g in G]
    q = [np.einsum("im,cmjk->cijk", D, u), np.einsum("jm,cimk->cijk", D, u), np.einsum("km,cijm->cijk", D, u)]
    v = [sum(G[g] * a for g, a in zip(r, q)) for r in ROWS]
    return np.einsum("mi,cmjk->cijk", D, v[0]) + np.einsum("mj,cimk->cijk", D, v[1]) + \
        np.einsum("mk,cijm->cijk", D, v[2])


def values(kind, shape, rng):
    w, t = rng.uniform(-1, 1, shape), np.linspace(0, 1, shape[1])
    if kind == "wide":
        return w * 2.0 ** (-60 * rng.random(shape))
    if kind == "offset":
        return 1 + 1e-6 * w
    c = [rng.uniform(-1, 1, (shape[0], 1, 1, 1)) for _ in range(4)]
    return np.sin(3 * c[0] + 0.1 * (c[1] * t[:, None, None] + c[2] * t[:, None] + c[3] * t)) + 1e-6 * w


@extended
def test_sums_on_the_grid_of_magnitudes_are_exact():
    x = np.random.default_rng(1).uniform(-1, 1, 4096).astype(f32)
    x[:2] = 1 - 2.0 ** -24, -(1 - 2.0 ** -24)
    h = np.copysign((f32(1) + np.abs(x)).astype(f32) - f32(1), x)
    for s in (1, -1):
        exactly = h[:, None].astype(EXT) + s * h[None, :].astype(EXT)
        assert np.array_equal((h[:, None] + f32(s) * h[None, :]).astype(EXT), exactly)
    assert np.abs(x - h).max() <= 2.0 ** -24


@extended
@pytest.mark.gpu
@pytest.mark.parametrize("p", range(1, 9))
@pytest.mark.parametrize("kind", ["wide", "offset", "smooth"])
def test_error_is_no_larger_than_the_plain_forms(p, kind):
    import torch

    import benchmarks_gb300 as mf
    n = p + 1
    rng = np.random.default_rng(p)
    D = gll_derivative(n)[1]
    D = 0.5 * (D - D[::-1, ::-1])
    shape = (1200 // n ** 2 + 20, n, n, n)
    G = [(0.2 * rng.random(shape) + (g in (0, 3, 5))) / 2.4 for g in range(6)]
    u = values(kind, shape, rng)
    u *= 2.0 ** -(np.floor(np.log2(np.abs(u).max(axis=(1, 2, 3), keepdims=True))) + 1)
    want = exact(D, u, G)
    y = plain(D, u, [split(g) for g in G])
    bound = np.sqrt(((y[0].astype(EXT) + y[1] - want) ** 2).sum())
    dev = [torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda() for a in (D, np.stack(G, axis=1), u)]
    got = mf.bk5_evector(p, *dev, torch.zeros_like(dev[2]), arith="df").cpu().numpy().reshape(shape)
    assert np.sqrt(((got - want) ** 2).sum()) <= bound
