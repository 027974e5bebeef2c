"""The FP64 reciprocal root of every FP64 sum (rinv_cut, kernels_common.cuh)
against 1 / sqrt(x) in extended precision and against CUDA's rsqrt().

Bound: with the seed's relative error d and e = 1 - x y^2 (|e| <= 2.1 d), the
truncated series leaves 5 e^3 / 16 < 3e-18 relative for d <= 1e-6; x y rounds by
2^-53, which moves e by as much and the result by 2^-54; the last operation
rounds by half a unit.  In units in the last place of a result between 1 and 2
times a power of two: 0.5 + 0.5 + 0.03, so 1.03; rsqrt() is within 1 of the
exact value, so within 2.03, hence 2 representable numbers, of this one.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUT = 1e-16


def _map(harness, which, x):
    x = np.ascontiguousarray(x, np.float64)
    y = np.zeros_like(x)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    assert harness.harness_root(which, p(x), len(x), p(y)) == 0
    return y


def _values():
    rng = np.random.default_rng(1)
    n = 1 << 20
    parts = [np.exp(rng.uniform(np.log(CUT), np.log(1e2), n)), np.exp(rng.uniform(np.log(CUT), 709.7, n)),
             1 + rng.uniform(0, 3, n)]  # one period of the root
    e = np.ldexp(1.0, np.arange(-53, 1024))
    parts += [e, np.nextafter(e, np.inf), np.nextafter(e, 0), [CUT, np.nextafter(CUT, 1), np.finfo(np.float64).max]]
    x = np.concatenate(parts)
    return x[(x >= CUT) & np.isfinite(x)]


def test_root_is_within_its_bound(gpu, harness):
    x = _values()
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    seed = np.abs(_map(harness, 1, x) / exact - 1)
    assert float(seed.max()) <= 1e-6
    got = _map(harness, 0, x)
    ulp = np.spacing(exact.astype(np.float64)).astype(np.longdouble)
    assert float(np.max(np.abs(got - exact) / ulp)) <= 1.03
    assert np.max(np.abs(got.view(np.int64) - _map(harness, 2, x).view(np.int64))) <= 2


def test_root_beyond_its_range_is_zero(gpu, harness):
    x = np.array([0.0, -0.0, 1e-320, 1e-17, np.nextafter(CUT, 0), np.inf, np.nan, -np.nan, -1.0, -np.inf])
    assert np.array_equal(_map(harness, 0, x), np.zeros(len(x)))
