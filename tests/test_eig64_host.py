"""Shared memory of the FP64 eigensolver up to the 4096 bands a model may have (no
GPU needed)."""

import ctypes

import pytest

from rustb_gb300 import _lib


@pytest.mark.parametrize("n", [9, 32, 33, 64, 65, 112, 113, 163, 164, 256, 512, 1024, 2048, 3000, 4096])
def test_fits_one_cta(n):
    fn = _lib.load().tbg_internal_eig64_smem
    fn.restype, fn.argtypes = ctypes.c_int64, [ctypes.c_int]
    # 227 KB per CTA, of which the panel kernel has up to 10 KB of static memory
    assert 0 < fn(n) <= (227 - (10 if n > 163 and fn(n) == 48 * n else 0)) * 1024
