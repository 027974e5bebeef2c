"""Evaluations at every accuracy without its own transform kernels (np = 2, 3, 5
and 7: cyclic grids of 3, 5, 9 and 13 points) and, beside them, np = 4, against
the method written out in NumPy for one level of 64 leaves: the check potentials
of the surfaces, a dense kernel matrix for every pair of the V list and the direct
sum of the neighbours.  The truncated pseudo-inverses are the library's own (two
LAPACK drivers alone move the result by 2e-10 at np = 7: the subspace that is cut
off is that ill-determined).

Tolerance: the pseudo-inverses magnify a rounding error along a direction of
singular value s by 1 / s, and the far evaluation damps that direction by about s
again, so a value keeps the rounding of its sums of about 4,000 terms, 2^-53 sqrt(4000)
times a small factor, 1e-13 to 1e-12; 1e-10 here.  Mixed precision: 2e-5, as the
mixed contractions' test.  The method itself is off by 10^-2 (np = 2) to 10^-7
(np = 7), so that agreement with the direct sum would show less.
"""
import ctypes

import numpy as np
import pytest

import kifmm
import workloads as W

pytestmark = pytest.mark.gpu


def _surface(p, radius):
    g = np.linspace(-1, 1, p)
    q = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return q[np.abs(q).max(1) > 1 - 1e-9] * radius


def _laplace(trg, src):
    r = np.linalg.norm(trg[:, None] - src[None], axis=2)
    return np.where(r < 1e-8, 0.0, 1 / (4 * np.pi * np.where(r < 1e-8, 1.0, r)))


def _pinv(harness, a, cut):
    m, n = a.shape
    a, v, w = np.ascontiguousarray(a), np.zeros(n * min(m, n)), np.zeros(m * min(m, n))
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    r = harness.harness_pinv(m, n, p(a), ctypes.c_double(cut), p(v), p(w))
    assert r > 0
    v, w = v[:n * r].reshape(n, r), w[:r * m].reshape(r, m)
    return lambda x: v @ (w @ x)


def _one_level(harness, src, trg, den, np_):
    h = 0.25  # radius of a leaf of depth 2
    ue, uc, de, dc = (_surface(p, r * h) for p, r in ((np_, 1), (np_ + 2, 3), (np_, 3), (np_, 1)))
    cut = 0.1 ** (np_ + 1)
    up, dn = _pinv(harness, _laplace(uc, ue), cut), _pinv(harness, _laplace(dc, de), cut)
    cells = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    ctr = -1 + h * (2 * cells + 1)
    of = lambda x: np.ravel_multi_index(np.minimum(((x + 1) / (2 * h)).astype(int), 3).T, (4, 4, 4))
    s, t = of(src), of(trg)
    q = [up(_laplace(uc + c, src[s == k]) @ den[s == k]) for k, c in enumerate(ctr)]
    out = np.zeros(len(trg))
    for k, c in enumerate(ctr):
        mine = trg[t == k]
        near = np.abs(cells - cells[k]).max(1) <= 1
        u = _laplace(mine, src[near[s]]) @ den[near[s]]
        check = sum(_laplace(dc + c, ue + ctr[j]) @ q[j] for j in range(64) if not near[j])
        out[t == k] = u + _laplace(mine, de + c) @ dn(check)
    return out


@pytest.mark.parametrize("np_", [2, 3, 4, 5, 7])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_level_matches_the_dense_method(gpu, harness, np_, precision):
    src, trg = W.cube(3000, 3)[0], W.cube(2000, 4)[0]
    den = W.densities(3000, 1, "uniform", 5)
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, src, trg
    f.knl = kifmm.Kernel3d(111, [1.0])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": "5", "-fmm3d_let3d_maxlevel": "3",
             "-fmm3d_precision": precision})
    t = f.tree()
    leaf = t["chd"] < 0
    assert t["maxdepth"] == 2 and leaf.sum() == 64
    out = np.zeros(2000)
    f.eval(den, out)
    want = _one_level(harness, src, trg, den, np_)
    assert np.linalg.norm(out - want) <= (1e-10 if precision == "fp64" else 2e-5) * np.linalg.norm(want)
