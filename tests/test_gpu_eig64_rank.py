"""FP64 eigensolver on rank-deficient matrices, whose reduction meets columns of
rounding errors of rounding errors down to the end of FP64's range, and on matrices
scaled towards its ends, with the bounds of test_gpu_eig64 (GPU)."""

import numpy as np
import pytest

from test_gpu_eig64 import check, random_hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 10, 16, 20, 25, 32, 33, 40, 47, 64, 65, 96, 112, 113, 128, 160, 164, 170, 200])
def test_rank_deficient(n):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    w = np.exp(2j * np.pi * np.arange(n) / n)[:, None]
    ones = np.ones((n, n), complex)
    check(np.stack([ones, 7.0 * ones, v @ v.conj().T, w @ w.conj().T, v[:, :1] @ v[:, :1].conj().T + np.eye(n),
                    np.outer(np.arange(n), np.arange(n)) + 0j]))


@pytest.mark.parametrize("n", [12, 40, 100, 170])
@pytest.mark.parametrize("scale", [1e-290, 1e-170, 1e-160, 1e-155, 1e155, 1e160, 1e200, 1e290])
def test_scaled(n, scale):
    check(random_hermitian(np.random.default_rng(n), 3, n) * scale)


@pytest.mark.parametrize("n", [20, 47, 64, 96, 128, 164, 200])
@pytest.mark.parametrize("spread", [1e-15, 1e-14, 1e-12, 1e-10])
def test_clusters_below_the_shifts(n, spread):
    """Eigenvalues nearer than the shifts of the inverse iteration can tell apart."""
    H = []
    for seed in range(4):
        rng = np.random.default_rng(seed)
        h = random_hermitian(rng, 1, n)[0]
        Q, _ = np.linalg.qr(h + 1j * np.eye(n))
        H += [np.ones((n, n)) + spread * h, (Q * (np.arange(n) // (n // 2) + 1.0)) @ np.conj(Q.T) + spread * h]
    H = np.stack(H)
    check(0.5 * (H + np.conj(np.transpose(H, (0, 2, 1)))))
