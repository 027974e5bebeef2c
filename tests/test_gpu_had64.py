"""The FP64 V-list Hadamard on matrix instructions against the direct
parent-pair sweep (-fmm3d_m2l_form direct), over its dispatch: the three dof
blocks, np 4, 6 and 8, one group of parents and a few rows of padding, more
parents than one sorting window (4,096; the volume of 40,000 points), volumes (every direction) and
surfaces (few), and several density vectors.

Both forms sum the same FP64 products in another order, with one more rounded
difference per operator value: a few hundred to a few thousand terms of
comparable size, relative 2^-53 * sqrt(3000) * 8 < 1e-13 per spectrum, damped
by the translation back to the points; 1e-12 as for the other pairs of forms.
"""
import numpy as np
import pytest

import kifmm
import workloads as W

pytestmark = pytest.mark.gpu


def _eval(kt, np_, src, nor, trg, den, ptsmax, nrhs, form):
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, nor, trg
    f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
    o = {"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": str(ptsmax), "-fmm3d_let3d_maxlevel": "10"}
    if form:
        o["-fmm3d_m2l_form"] = form
    f.setup(o)
    if len(src) == 40000:  # target parents of the V list: more than one window of 4,096
        t = f.tree()
        assert len(set(t["par"][np.diff(t["V_ptr"]) > 0])) > 4096
    out = np.zeros((nrhs, f.tdof() * len(trg)))
    f.eval_multi(den.reshape(nrhs, -1), out)
    return out


@pytest.mark.parametrize("kt", [111, 321, 511])
@pytest.mark.parametrize("np_,geometry,n,ptsmax,nrhs", [
    (4, "sphere", 300, 20, 1), (4, "cube", 30000, 4, 1), (6, "ellipsoid", 3001, 30, 2), (6, "plummer_ball", 4000, 40, 1),
    (8, "sphere", 1500, 60, 1), (4, "cube", 40000, 4, 1), (6, "cube", 40000, 4, 1)])
def test_matrix_hadamard_matches_direct_sweep(gpu, kt, np_, geometry, n, ptsmax, nrhs):
    src, nor = W.GEOMETRIES[geometry](n, 3)
    trg = W.cube(n // 3, 4)[0] if n == 3001 else src
    den = W.densities(n * nrhs, kifmm.Kernel3d.DOFS[kt][0], "uniform", 5)
    got = _eval(kt, np_, src, nor, trg, den, ptsmax, nrhs, None)
    want = _eval(kt, np_, src, nor, trg, den, ptsmax, nrhs, "direct")
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
