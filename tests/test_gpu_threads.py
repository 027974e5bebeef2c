"""Two handles evaluated by two threads at once, as include/kifmm.h allows for
distinct handles.  Kernels that both use take different amounts of dynamic
shared memory: the surface contractions by the size of a level, the tensor-core
Hadamard by the size of the tree, the inverse transform by the V-list form, the
transforms of np other than 4, 6 and 8 by np.

Every eval has to succeed and, an evaluation being deterministic, to return
the bits that the same handle returns alone.
"""
import threading

import numpy as np
import pytest

import kifmm
import workloads as W

pytestmark = pytest.mark.gpu


def _handle(n, np_, precision, form, seed):
    src = W.cube(n, seed)[0]
    f = kifmm.FMM3d("fmm3d_")
    f.srcpos, f.srcnor, f.trgpos = src, src, src
    f.knl = kifmm.Kernel3d(111, [1.0])
    f.setup({"-fmm3d_np": str(np_), "-fmm3d_let3d_ptsmax": "5", "-fmm3d_let3d_maxlevel": "10",
             "-fmm3d_precision": precision, "-fmm3d_m2l_form": form})
    return f, W.densities(n, 1, "uniform", seed + 1)


@pytest.mark.parametrize("precision,forms,nps", [("fp64", ("toeplitz", "toeplitz"), (4, 4)),
                                                 ("fp64", ("direct", "direct"), (3, 5)),
                                                 ("mixed", ("tensor", "tensor"), (4, 4)),
                                                 ("mixed", ("tensor", "toeplitz"), (4, 4))])
def test_two_handles_from_two_threads(gpu, precision, forms, nps):
    torch = pytest.importorskip("torch")
    jobs = []
    for k, n in enumerate((3000, 20000)):
        f, den = _handle(n, nps[k], precision, forms[k], 1 + k)
        d_den, d_out = torch.from_numpy(den).cuda(), torch.zeros(n, device="cuda", dtype=torch.float64)
        f.eval_device(d_den.data_ptr(), d_out.data_ptr(), 1, 0, sync=True)
        jobs.append((f, d_den, d_out, d_out.clone(), torch.cuda.Stream()))
    torch.cuda.synchronize()
    start, bad = threading.Barrier(2), []

    def run(k):
        f, d_den, d_out, want, stream = jobs[k]
        start.wait()
        for i in range(1500):
            try:
                f.eval_device(d_den.data_ptr(), d_out.data_ptr(), 1, stream.cuda_stream, sync=True)
            except kifmm.KifmmError as e:
                bad.append((k, i, str(e)))
                return
            if not torch.equal(d_out, want):
                bad.append((k, i, "another result"))
                return

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not bad, bad
