"""X lists: target nodes on a densely refined surface with the coarse source
leaves of a sparse volume beside them, so that their downward check surfaces take
whole lists of source leaves (S2L), at np whose check points fill one to ten
blocks of 32 and lists below and above 128 leaves.

Against the direct sum: the np = 4 and 6 expansions truncate below 5e-3 and 2e-4 on
the committed fixtures, np = 8 below 1e-5; a lost leaf or check point costs
percents of the near field.
"""
import numpy as np
import pytest

import kifmm
import oracle
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,precision", [(111, "fp64"), (111, "mixed"), (321, "mixed"), (511, "fp64")])
@pytest.mark.parametrize("np_,bound", [(4, 1e-2), (6, 1e-3), (8, 1e-4)])
def test_fine_targets_beside_coarse_sources(gpu, kt, precision, np_, bound):
    trg, _ = W.ellipsoid(20000, 3)
    sph, sn = W.sphere(6000, 8)
    cub = W.cube(3000, 4)[0] * 0.999
    src = np.concatenate([cub, sph * 0.3])
    nor = np.concatenate([cub, sn])
    den = W.densities(len(src), kifmm.Kernel3d.DOFS[kt][0], "uniform01", 5)
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, nor, trg
    f.knl = kifmm.Kernel3d(kt, [1.0, 0.3])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": "15", "-fmm3d_let3d_maxlevel": "10",
             "-fmm3d_precision": precision})
    t = f.tree()
    assert (np.diff(t["X_ptr"]) > 0).any()
    out = np.zeros(f.tdof() * len(trg))
    f.eval(den, out)
    idx = W.check_indices(len(trg), 500)
    want = oracle.direct(kt, [1.0, 0.3], src, nor, den, trg[idx])
    got = out.reshape(len(trg), -1)[idx].ravel()
    assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want)
