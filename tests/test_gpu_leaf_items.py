"""The leaf pass's work items at the edges of their cuts: one leaf whose
source range is cut inside a source leaf, rounds of 1 to 32 targets, and
coarse target leaves whose W lists hold many surfaces, in FP64 and (mixed)
FP32 with the FP64 near field of double layers.

Trees of depth 0 and 1 have no far field, so the evaluation is the direct sum:
in FP64 the relative error stays below sqrt(n) * 10 * 2^-53 < 1e-13 (1e-12
here); in mixed precision the coordinates' 2^-24 dominates a single layer's
terms (nearest neighbours: leaf size over distance, up to a few hundred), 1e-4;
the double layers' near field is FP64 with the FP32 rounding of nothing else.
"""
import numpy as np
import pytest

import kifmm
import oracle
import workloads as W

pytestmark = pytest.mark.gpu


def _run(kt, src, nor, trg, den, np_, ptsmax, maxlevel, precision):
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, nor, trg
    f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": str(ptsmax), "-fmm3d_let3d_maxlevel": str(maxlevel),
             "-fmm3d_precision": precision})
    out = np.zeros(len(trg) * f.tdof())
    f.eval(den, out)
    return out


@pytest.mark.parametrize("kt,precision,tol", [(111, "fp64", 1e-12), (311, "fp64", 1e-12), (321, "fp64", 1e-12),
                                              (111, "mixed", 1e-4), (121, "mixed", 1e-12)])
@pytest.mark.parametrize("ns,nt", [(1, 1), (63, 31), (129, 33), (5000, 1), (5000, 32), (5001, 65)])
@pytest.mark.parametrize("ptsmax", [10 ** 6, 40])
def test_cut_ranges_are_the_direct_sum(gpu, kt, precision, tol, ns, nt, ptsmax):
    src, nor = W.ellipsoid(ns, 3)
    trg = W.cube(nt, 4)[0]
    den = W.densities(ns, kifmm.Kernel3d.DOFS[kt][0], "uniform", 5)
    got = _run(kt, src, nor, trg, den, 4, ptsmax, 1, precision)
    want = oracle.direct(kt, [1.0, 0.3], src, nor, den, trg)
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("kt,precision", [(111, "fp64"), (121, "mixed"), (311, "mixed")])
def test_coarse_targets_with_long_w_lists(gpu, kt, precision):
    """np = 6 truncates at about 1e-5 (every committed np = 6 fixture is below 2e-4);
    a dropped surface or source leaf costs percents."""
    src, nor = W.ellipsoid(30000, 3)
    trg = W.cube(700, 4)[0] * 0.999
    den = W.densities(30000, kifmm.Kernel3d.DOFS[kt][0], "uniform01", 5)
    got = _run(kt, src, nor, trg, den, 6, 60, 10, precision)
    want = oracle.direct(kt, [1.0, 0.3], src, nor, den, trg)
    assert np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want)
