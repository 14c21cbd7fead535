"""Reciprocal and reciprocal square root of the FP64 solver against numpy's (GPU).

The residual e of the hardware's approximation is below 2^-19, so the step's error term
e^3 is below 2^-57 and the rounding of the last operation (half a unit in the last
place) with those of e and of the correction leaves at most one unit in all; the
square root's residual has one rounding more, in x y."""

import ctypes

import numpy as np
import pytest

from rustb_gb300 import _lib

pytestmark = pytest.mark.gpu


def test_units_in_the_last_place():
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.uniform(1, 4, 200000) * 2.0 ** rng.integers(-900, 900, 200000),
                        1.0 + np.arange(-2000, 2000) * np.finfo(float).eps, 2.0 - np.arange(2000) * 2.0 ** -52,
                        2.0 ** np.arange(-1000.0, 1000.0)])
    x *= rng.choice([-1.0, 1.0], x.size)
    lib = _lib.load()
    dp = ctypes.POINTER(ctypes.c_double)
    fn = lib.tbg_internal_fast_math
    fn.restype, fn.argtypes = ctypes.c_int, [ctypes.c_int, dp, dp, dp]
    r, s = np.empty_like(x), np.empty_like(x)
    _lib.check(fn(x.size, *(a.ctypes.data_as(dp) for a in (x, r, s))), lib)
    lx = x.astype(np.longdouble)
    for got, ref, ulps in ((r, 1 / lx, 1.0), (s, 1 / np.sqrt(abs(lx)), 1.5)):
        ulp = np.spacing(np.abs(ref.astype(float)))
        assert np.max(np.abs(got - ref) / ulp) <= ulps
