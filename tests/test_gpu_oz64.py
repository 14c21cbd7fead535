"""FP64-accurate tensor-core products against numpy (GPU).

A value is kept to 2^-56 of its line's power of two and the dropped digit pairs
are of the same size, so a contraction of K complex terms is within
4 (K + 8) 2^-54 of (line of A's largest) x (column of B's largest) x 4 (the line
exponents round up by less than 2 each)."""

import ctypes

import numpy as np
import pytest

from rustb_gb300 import _lib

pytestmark = pytest.mark.gpu


def gemm(A, B, C, conj_a, conj_b, mode):
    lib = _lib.load()
    dp = ctypes.POINTER(ctypes.c_double)
    fn = lib.tbg_internal_oz64_gemm
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int64] + [ctypes.c_int] * 4 + [dp] * 3
    out = np.ascontiguousarray(C).copy()
    Ac, Bc = np.ascontiguousarray(A), np.ascontiguousarray(B)
    M, K = (A.shape[2], A.shape[1]) if conj_a else (A.shape[1], A.shape[2])
    Nc = B.shape[1] if conj_b else B.shape[2]
    ptr = lambda x: x.view(np.float64).ctypes.data_as(dp)  # noqa: E731
    _lib.check(fn(int(conj_a), int(conj_b), A.shape[0], M, Nc, K, mode, ptr(Ac), ptr(Bc), ptr(out)), lib)
    return out


def case(batch, M, Nc, K, conj_a, conj_b, seed):
    rng = np.random.default_rng(seed)
    z = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    A = z(batch, M, K) * 10.0 ** rng.uniform(-30, 30, (batch, M, 1))
    B = z(batch, K, Nc) * 10.0 ** rng.uniform(-30, 30, (batch, 1, Nc))
    ref = np.einsum("bmk,bkn->bmn", A.astype(np.clongdouble), B.astype(np.clongdouble))
    scale = (np.abs(A).max(2)[:, :, None] * np.abs(B).max(1)[:, None, :])
    stored = lambda x, c: np.conj(x.transpose(0, 2, 1)) if c else x  # noqa: E731
    return stored(A, conj_a), stored(B, conj_b), ref, scale


@pytest.mark.parametrize("conj_a,conj_b", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("batch,M,Nc,K", [(1, 1, 1, 1), (3, 128, 128, 128), (400, 33, 33, 33), (2, 129, 49, 17),
                                          (5, 64, 64, 64), (2, 200, 97, 256), (1, 130, 31, 600)])
def test_products(batch, M, Nc, K, conj_a, conj_b):
    A, B, ref, scale = case(batch, M, Nc, K, conj_a, conj_b, M + Nc + K)
    tol = 16.0 * (K + 8) * 2.0 ** -54 * scale
    C0 = np.ones_like(ref, dtype=complex) * scale
    got = gemm(A, B, C0, conj_a, conj_b, 0)
    assert np.all(np.abs(got - ref) <= tol)
    sub = gemm(A, B, C0, conj_a, conj_b, -1)
    assert np.all(np.abs(sub - (C0 - ref)) <= 2 * tol)


def test_error_no_larger_than_fp64():
    A, B, ref, scale = case(20, 128, 128, 128, 0, 0, 5)
    oz = np.abs(gemm(A, B, np.zeros_like(A), 0, 0, 0) - ref) / scale
    fp = np.abs(A @ B - ref) / scale
    assert oz.max() <= fp.max()


def test_special_values():
    A, B, ref, scale = case(2, 40, 50, 20, 0, 0, 9)
    A[0, 3] = 0.0
    A[1, 7, 2] = np.nan
    B[1, 4, 11] = np.inf
    B[0, :, 5] = 3e-310
    got = gemm(A, B, np.zeros((2, 40, 50), complex), 0, 0, 0)
    assert np.all(got[0, 3] == 0.0)
    assert not np.any(np.isfinite(got[1, 7])) and not np.any(np.isfinite(got[1, :, 11]))
    ok = np.ones((2, 40, 50), bool)
    ok[1, 7], ok[1, :, 11], ok[0, 3], ok[0, :, 5] = False, False, False, False
    assert np.all(np.abs(got - ref)[ok] <= 1e-12 * scale[ok])
