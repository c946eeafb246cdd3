"""The h-prolongation's weights in FP32: every one is the FP64 product of its three axis
weights, rounded once, also where two or three axes end in a narrower coarse cell.
The node function runs on the host, on unit vectors (a result is then one weight)."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "mfgb_mg_kernels.cuh"
using namespace mfgb;
double mfgb::lagrange_value(int, const double *, int, double) { return 0; }  // (p-transfers: not used)
int main(int, char **a) {
  const int nx = atoi(a[1]), ny = atoi(a[2]), nz = atoi(a[3]), s = atoi(a[4]);
  auto cells = [](int n, int s) { return (n + s - 1) / s; };
  const HGrid g{cells(nx, s) + 1, cells(ny, s) + 1, cells(nz, s) + 1, cells(nx, 2 * s) + 1,
                cells(ny, 2 * s) + 1, cells(nz, 2 * s) + 1, {nx, ny, nz}, s};
  const int nf = g.fx * g.fy * g.fz, nc = g.cx * g.cy * g.cz;
  std::vector<float> f(nf), c(nc);
  auto row = [](const std::vector<float> &v) { fwrite(v.data(), 4, v.size(), stdout); };
  for (int i = 0; i < nc; ++i) {
    std::fill(c.begin(), c.end(), 0.f), std::fill(f.begin(), f.end(), 0.f);
    c[i] = 1.f;
    for (int t = 0; t < nf; ++t) h_prolongate_node(g, t, c.data(), f.data());
    row(f);
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from benchmarks_gb300 import build
    d = tmp_path_factory.mktemp("h")
    src, exe = d / "h.cu", d / "h"
    src.write_text("#include <vector>\n" + PROGRAM)
    subprocess.run([build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-I" + build.CSRC,
                    "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True, timeout=600)
    return str(exe)


def axis(n, s):
    """FP64 interpolation [fine node, coarse node] of one axis; nodes at min(k s, n)"""
    fine = [min(k * s, n) for k in range(-(-n // s) + 1)]
    coarse = [min(2 * k * s, n) for k in range(-(-n // (2 * s)) + 1)]
    P = np.zeros((len(fine), len(coarse)))
    for i, x in enumerate(fine):
        if i % 2 == 0:
            P[i, i // 2] = 1
        else:
            lo, hi = coarse[i // 2], coarse[i // 2 + 1]
            r = (x - lo) / (hi - lo)
            P[i, i // 2], P[i, i // 2 + 1] = 1 - r, r
    return P


@pytest.mark.parametrize("n,s", [((4, 6, 8), 1), ((7, 5, 3), 1), ((7, 11, 13), 2), ((11, 8, 13), 2), ((23, 13, 21), 4)])
def test_weights_are_products_rounded_once(program, n, s):
    out = np.frombuffer(subprocess.run([program, *map(str, n), str(s)], capture_output=True, check=True,
                                       timeout=300).stdout, dtype=np.float32)
    Px, Py, Pz = (axis(m, s) for m in n)
    fine, coarse = Px.shape[0] * Py.shape[0] * Pz.shape[0], Px.shape[1] * Py.shape[1] * Pz.shape[1]
    W = np.einsum("zc,yb,xa->zyxcba", Pz, Py, Px)
    inside = np.zeros(W.shape[:3], dtype=bool)
    inside[1:-1, 1:-1, 1:-1] = True
    W = W.reshape(fine, coarse).astype(np.float32)
    assert np.array_equal(out.reshape(coarse, fine), np.where(inside.reshape(-1), W.T, 0))
