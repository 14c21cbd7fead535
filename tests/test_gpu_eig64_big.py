"""The FP64 eigensolver beyond one SM's shared memory (a cluster of CTAs per
matrix, digit products for the updates) and the blocked back-transformation, with
the bounds of test_gpu_eig64 (GPU)."""

import numpy as np
import pytest

from test_gpu_eig64 import check, random_hermitian
from rustb_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(165, 1), (177, 40), (192, 2), (193, 160), (256, 3), (257, 2), (300, 9), (512, 2),
                                  (56, 260), (63, 180), (65, 170), (97, 60), (128, 24), (129, 30), (161, 12)])
def test_random(n, nk):
    check(random_hermitian(np.random.default_rng(n), nk, n))


@pytest.mark.parametrize("n", [166, 258])
def test_degenerate_scaled_and_split(n):
    rng = np.random.default_rng(n)
    b = random_hermitian(rng, 1, n // 2)[0]
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    z = np.zeros_like(b)
    H = random_hermitian(rng, 1, n)[0]
    tri = np.diag(np.arange(n) % 3 + 0.0) + np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1)
    mats = [Q @ np.block([[b, z], [z, b]]) @ np.conj(Q.T), Q @ np.diag((np.arange(n) % 3) * 1.0) @ np.conj(Q.T),
            np.block([[b, z], [z, 2 * b]]), H.real + 0j, tri + 0j, np.diag(np.arange(n) - 7.0) + 0j, H * 1e-120, H * 1e120]
    H = np.stack(mats)
    check(0.5 * (H + np.conj(np.transpose(H, (0, 2, 1)))))


@pytest.mark.parametrize("n,nk", [(100, 3), (170, 5), (200, 170), (400, 30)])
def test_values_only(n, nk):
    m = W.random_model(2, n, False, 1, seed=n)
    k = np.random.default_rng(n).uniform(0, 1, (nk, 2))
    H = m.gen_ham_batch(k)
    E = m.solve_band_all_parallel(k)
    ref = np.linalg.eigvalsh(H)
    assert np.all(np.diff(E, axis=1) >= 0)
    assert np.max(np.abs(E - ref)) <= 16 * n * np.finfo(float).eps * np.max(np.abs(ref))
