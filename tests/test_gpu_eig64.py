"""The FP64 eigensolver (reduction, tridiagonal stage, back-transformation) on
its own, against LAPACK's eigenvalues and by residual and orthogonality (GPU).

Bounds: Householder reduction and back-transformation are backward stable with
a constant of a few N eps ||H|| (16 N eps taken).  Two vectors from the twisted
factorisation are formed independently when their eigenvalues lie at least
1e-3 ||T|| apart, each with a backward error of about 4 eps ||T||, so their
inner product stays below 2 * 4 eps / 1e-3 = 1.8e-12, to which the reflectors
add a few N eps."""

import ctypes

import numpy as np
import pytest

from rustb_gb300 import _lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def eig_f64(H):
    lib = _lib.load()
    nk, n = H.shape[0], H.shape[1]
    E = np.zeros((nk, n))
    U = np.zeros((nk, n, n), dtype=np.complex128)
    dp = ctypes.POINTER(ctypes.c_double)
    fn = lib.tbg_internal_eig_f64
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_int, ctypes.c_int64, dp, dp, dp, ctypes.c_int, ctypes.c_int,
                   ctypes.POINTER(ctypes.c_float)]
    H = np.ascontiguousarray(H, dtype=np.complex128)
    ms = ctypes.c_float(0.0)
    _lib.check(fn(n, nk, H.view(np.float64).ctypes.data_as(dp), E.ctypes.data_as(dp),
                  U.view(np.float64).ctypes.data_as(dp), 0, 1, ctypes.byref(ms)), lib)
    return E, U


def check(H):
    E, U = eig_f64(H)
    n = H.shape[1]
    nrm = np.maximum(np.linalg.norm(H, 2, axis=(1, 2)), 1e-300)
    tol = 16 * n * EPS
    assert np.all(np.diff(E, axis=1) >= 0)
    assert np.max(np.abs(E - np.linalg.eigvalsh(H)) / nrm[:, None]) <= tol
    assert np.max(np.abs(H @ U - U * E[:, None, :]).max(axis=(1, 2)) / nrm) <= tol
    assert np.max(np.abs(np.conj(np.transpose(U, (0, 2, 1))) @ U - np.eye(n))) <= 2e-12 + tol


def random_hermitian(rng, nk, n):
    X = rng.standard_normal((nk, n, n)) + 1j * rng.standard_normal((nk, n, n))
    return 0.5 * (X + np.conj(np.transpose(X, (0, 2, 1))))


@pytest.mark.parametrize("n,nk", [(9, 1), (9, 1300), (14, 37), (16, 9), (17, 5), (31, 8), (32, 1231), (33, 40), (48, 3),
                                  (64, 170), (65, 4), (97, 3), (112, 2), (113, 3), (128, 5), (150, 2), (161, 2),
                                  (163, 2)])
def test_random(n, nk):
    check(random_hermitian(np.random.default_rng(n), nk, n))


@pytest.mark.parametrize("n", [10, 20, 32, 34, 66, 130])
def test_degenerate_scaled_and_split(n):
    """Pairwise degenerate spectra, a few-level spectrum, decoupled blocks, a
    real matrix, one already tridiagonal, and extreme scales."""
    rng = np.random.default_rng(n)
    b = random_hermitian(rng, 1, n // 2)[0]
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    z = np.zeros_like(b)
    H = random_hermitian(rng, 1, n)[0]
    tri = np.diag(np.arange(n) % 3 + 0.0) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    mats = [Q @ np.block([[b, z], [z, b]]) @ np.conj(Q.T), Q @ np.diag((np.arange(n) % 3) * 1.0) @ np.conj(Q.T),
            np.block([[b, z], [z, 2 * b]]), H.real + 0j, tri + 0j, H * 1e-120, H * 1e120]
    H = np.stack(mats)
    check(0.5 * (H + np.conj(np.transpose(H, (0, 2, 1)))))


@pytest.mark.parametrize("n", [12, 32, 40, 100])
def test_diagonal_is_exact(n):
    d = np.random.default_rng(n).standard_normal((2, n))
    E, _ = eig_f64(np.stack([np.diag(x) for x in d]) + 0j)
    assert np.array_equal(E, np.sort(d, axis=1))
