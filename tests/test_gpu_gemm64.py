"""The FP64 surface contractions at the shapes where their tiles end: every
np's surface and rank sizes (8 to 296 points times the dofs, both tile widths),
trees whose levels have fewer columns than one tile of 64 nodes (K split over a
cluster) and many, and the level-scaled epilogue of a shifted root level.

The evaluation is compared with the direct sum: the expansions truncate below
10^(2 - np) (the committed fixtures: 3e-4 at np = 4, 2e-4 at 6, 6e-8 at 8), while
a wrong tile, slice or row changes the far field itself.
"""
import numpy as np
import pytest

import kifmm
import oracle
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_", [3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("kt,n,ptsmax,rootlvl", [(111, 700, 10, 0), (111, 30000, 20, -1), (311, 4000, 40, 0),
                                                 (511, 3000, 60, 0)])
def test_contractions_reach_the_truncation_error(gpu, np_, kt, n, ptsmax, rootlvl):
    scale = 2.0 ** -rootlvl
    src = W.cube(n, 3)[0] * scale
    den = W.densities(n, kifmm.Kernel3d.DOFS[kt][0], "uniform", 5)
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, src, src
    f.rootlvl = rootlvl
    f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": str(ptsmax), "-fmm3d_let3d_maxlevel": "10"})
    out = np.zeros(n * f.tdof())
    f.eval(den, out)
    idx = W.check_indices(n, 300)
    want = oracle.direct(kt, [1.0, 0.3], src, src, den, src[idx])
    got = out.reshape(n, -1)[idx].ravel()
    assert np.linalg.norm(got - want) <= 10.0 ** (2 - np_) * np.linalg.norm(want)
