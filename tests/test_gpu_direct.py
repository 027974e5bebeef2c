"""The direct sum at the edges of its split: target counts around the 8, 32
and 128 targets of a block, source counts around one staged tile of 128, and
many chunks of sources, against the oracle's restatement of Dense3d::eval.

Tolerance: a sum of n FP64 terms of random sign keeps about sqrt(n) times the
size of one term, each term is exact to a few units in the last place and the
partial sums round n times at most, so the relative error stays below
sqrt(n) * 10 * 2^-53 < 1e-13 for n <= 6,000; 1e-12 leaves a factor of ten.
"""
import numpy as np
import pytest

import kifmm
import oracle
import workloads as W

pytestmark = pytest.mark.gpu


def _engine(kt, src, nor):
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, nor, src
    f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
    f.setup({"-fmm3d_np": "4", "-fmm3d_let3d_ptsmax": "100", "-fmm3d_let3d_maxlevel": "10"})
    return f


@pytest.mark.parametrize("kt", sorted(kifmm.Kernel3d.DOFS))
@pytest.mark.parametrize("ns", [1, 127, 129, 6000])
def test_direct_sum_edges(gpu, kt, ns):
    src, nor = W.ellipsoid(ns, 5)
    den = W.densities(ns, kifmm.Kernel3d.DOFS[kt][0], "uniform", 6)
    f = _engine(kt, src, nor)
    for nt in (1, 8, 9, 33, 255, 257):
        trg = W.cube(nt, 7)[0]
        trg[0] = src[0]  # a source at the target itself adds nothing
        got = f.direct(den, trg)
        want = oracle.direct(kt, [1.0, 0.3], src, nor, den, trg)
        assert np.linalg.norm(got - want) <= 1e-12 * max(np.linalg.norm(want), 1e-300), (kt, ns, nt)


def test_direct_sum_far_target(gpu):
    """A target so far that r^2 overflows gets 1/r = 0, not a NaN."""
    src, nor = W.sphere(200, 1)
    f = _engine(111, src, nor)
    out = f.direct(np.ones(200), np.array([[1e200, 0.0, 0.0], [2.0, 0.0, 0.0]]))
    assert out[0] == 0.0 and np.isfinite(out[1]) and out[1] > 0
