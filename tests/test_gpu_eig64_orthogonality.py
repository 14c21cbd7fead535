"""Orthogonality of the FP64 solver's vectors for spectra without clusters (GPU).

A vector of the twisted factorisation is formed at a shift that is off by half an eps
||T|| typically (one eps at most), which leaves it eps ||T|| / (2 gap) along a neighbour. n levels
of a random matrix have gaps of ||T|| / n and n such pairs, so the Frobenius norm of U^H U - 1
is about n^1.5 eps / 2 for a typical matrix; the median over matrices has to lie below."""

import numpy as np
import pytest

from test_gpu_eig64 import eig_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 33, 64, 97])
def test_median_orthogonality(n):
    rng = np.random.default_rng(n)
    H = rng.standard_normal((40, n, n)) + 1j * rng.standard_normal((40, n, n))
    H = H + np.conj(np.transpose(H, (0, 2, 1)))
    E, U = eig_f64(H)
    off = np.linalg.norm(np.conj(np.transpose(U, (0, 2, 1))) @ U - np.eye(n), axis=(1, 2))
    assert np.median(off) <= 0.5 * n ** 1.5 * np.finfo(float).eps
