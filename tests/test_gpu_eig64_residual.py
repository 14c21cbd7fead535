"""Residual of the FP64 solver's eigenpairs where the back-transformation runs in
blocks of reflectors on the tensor cores (GPU).

2 n reflectors act on every vector, each with an error of about eps of the vector in
a random direction: H U - U E is about sqrt(2 n) eps ||H|| in the Frobenius norm."""

import numpy as np
import pytest

from test_gpu_eig64 import eig_f64, random_hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(64, 200), (97, 60), (128, 30), (161, 14), (170, 12), (170, 24), (256, 4), (256, 8)])
def test_residual_of_blocked_reflectors(n, nk):
    H = random_hermitian(np.random.default_rng(n), nk, n)
    E, U = eig_f64(H)
    res = np.linalg.norm(H @ U - U * E[:, None, :], axis=(1, 2)) / np.linalg.norm(H, axis=(1, 2))
    assert np.max(res) <= np.sqrt(2.0 * n) * np.finfo(float).eps
