"""The mixed engine's surface contractions over their dispatch: levels of one
column to several hundred (mma.sync, K split over clusters of 1 to 8), launches
of as many 128-node tiles as the GPU has SMs (tcgen05), both tile widths, one and
three dofs, several density vectors per pass (columns times vectors).

Against the FP64 engine on the same tree: products carry 2^-21 and the spectra
2^-22 relative, and the committed mixed fixtures differ from FP64 by at most
4e-6 at np <= 6; 2e-5 here.  np = 8 adds the FP32 floor of its pseudo-inverse (2e-6
measured on the full-size configuration).
"""
import numpy as np
import pytest

import kifmm
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", [111, 311, 511])
@pytest.mark.parametrize("np_,geometry,n,ptsmax,nrhs", [(4, "cube", 200, 10, 1), (4, "cube", 120000, 6, 1),
                                                        (6, "sphere", 5000, 40, 3), (6, "cube", 60000, 8, 1),
                                                        (8, "ellipsoid", 3000, 60, 1)])
def test_mixed_contractions_match_fp64(gpu, kt, np_, geometry, n, ptsmax, nrhs):
    src, nor = W.GEOMETRIES[geometry](n, 3)
    den = W.densities(n * nrhs, kifmm.Kernel3d.DOFS[kt][0], "uniform", 5).reshape(nrhs, -1)
    out = {}
    for prec in ("mixed", "fp64"):
        f = kifmm.FMM3d("fmm3d_")
        f.srcpos, f.srcnor, f.trgpos = src, nor, src
        f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
        f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": str(ptsmax), "-fmm3d_let3d_maxlevel": "10",
                 "-fmm3d_precision": prec})
        out[prec] = np.zeros((nrhs, f.tdof() * n))
        f.eval_multi(den, out[prec])
    assert np.linalg.norm(out["mixed"] - out["fp64"]) <= 2e-5 * np.linalg.norm(out["fp64"])
