"""The node contractions alone, on random operators and columns, against NumPy
at their rounding: operator rows and inner sizes around the tiles' edges (64,
128 and 160 rows, 16 or 32 inner values), column counts around the 64 and 128
nodes of a tile, K split over clusters and not, more tiles than SMs, gathered
and scattered columns, accumulation, and the scaling by level and dof.

Bounds, per value against the sum of |a| |b| (plus what it is added to): in FP64
every product and addition rounds once, in any order, and NumPy's own sum as
often: 2 (K + 2) 2^-53.  In the split TF32 form an operand keeps 22 bits and the
tail times tail product is dropped, 3 x 2^-22; the 12 MMAs of 32 inner values fold
into one accumulator with a 2^-22 each at most, the chunks are added in FP32, and
the result is rounded: (3 + 12) 2^-22 + (K / 32 + 4) 2^-23.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(harness, dtype, M, K, ncol, accumulate, sd, levels, num_sms=148):
    rng = np.random.default_rng(M + 7 * K + 11 * ncol)
    A = rng.standard_normal((M, K))
    nb, ldb, nc, ldc = ncol + 5, K + 4, ncol + 3, M + 8
    B = rng.standard_normal((nb, ldb)).astype(dtype)
    C = rng.standard_normal((nc, ldc)).astype(dtype)
    bidx, cidx = rng.permutation(nb)[:ncol].astype(np.int32), rng.permutation(nc)[:ncol].astype(np.int32)
    deg = np.array([1, 2, 0, 1][:sd], np.int32)
    lvl = rng.integers(0, 6, ncol).astype(np.int32) if levels else None
    p = lambda a: None if a is None else a.ctypes.data_as(ctypes.c_void_p)
    got = C.copy()
    f = harness.harness_gemm64 if dtype == np.float64 else harness.harness_gemm32
    assert f(M, K, p(A), nb, ldb, p(B), p(bidx), nc, ldc, p(got), p(cidx), ncol, accumulate, sd, p(deg), p(lvl), -1,
             num_sms) == 0
    scale = np.ones((ncol, M))
    if levels:
        scale = 2.0 ** (-(lvl[:, None] - 1) * deg[np.arange(M) % sd][None, :])
    cols = B[bidx][:, :K].astype(np.float64)
    want = C.astype(np.float64)
    old = want[cidx, :M] if accumulate else 0.0
    want[cidx, :M] = scale * (cols @ A.T) + old
    size = np.abs(want) * 0
    size[cidx, :M] = scale * (np.abs(cols) @ np.abs(A).T) + np.abs(old)
    return got, want, size


SHAPES = [(2, 2), (8, 56), (56, 18), (62, 30), (64, 16), (66, 64), (98, 130), (152, 152), (160, 96), (162, 34), (222, 1216),
          (296, 296), (320, 128)]


@pytest.mark.parametrize("M,K", SHAPES)
@pytest.mark.parametrize("ncol", [1, 63, 64, 65, 700, 12000])
def test_fp64_contraction(gpu, harness, M, K, ncol):
    accumulate, levels = ncol % 2, ncol in (65, 700, 12000)
    sd = 3 if M % 3 == 0 else 4 if M % 8 == 0 else 1
    got, want, size = _run(harness, np.float64, M, K, ncol, accumulate, sd, levels)
    assert np.all(np.abs(got - want) <= 2 * (K + 2) * 2.0 ** -53 * size)


@pytest.mark.parametrize("M,K,ncols", [(M, K, (1, 63, 64, 65, 700)) for M, K in
                                       [(4, 8), (8, 56), (56, 20), (64, 32), (68, 64), (100, 132), (152, 152), (160, 96),
                                        (164, 36), (224, 1216), (296, 296)]] +
                         [(M, K, (20000,)) for M, K in  # tcgen05: surface and rank sizes of np = 4 to 8
                          [(56, 152), (64, 56), (152, 296), (160, 96), (224, 1216), (296, 296)]])
def test_split_tf32_contraction(gpu, harness, M, K, ncols):
    for ncol in ncols:
        accumulate, levels = ncol % 2, ncol in (65, 700, 20000)
        sd = 4 if M % 8 == 0 else 1
        got, want, size = _run(harness, np.float32, M, K, ncol, accumulate, sd, levels)
        tol = 15 * 2.0 ** -22 + (K / 32 + 4) * 2.0 ** -23
        assert np.all(np.abs(got - want) <= tol * size), ncol
