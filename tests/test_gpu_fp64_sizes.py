"""FP64 velocities, rotation and position-matrix term at the sizes where the
kernels change: band-resolved Berry curvature against the numpy oracle (GPU).

The tolerance is the FP64 path's: energies 1e-10 ||H||, Omega 1e-8 of its
largest value (relative gaps of these models leave a factor of 1e4 and more)."""

import numpy as np
import pytest

from oracle import tb_oracle as O
from rustb_gb300 import Parameters, workloads as W

pytestmark = pytest.mark.gpu


def with_rmatrix(m, seed):
    rng = np.random.default_rng(seed)
    n = m.nsta
    r = 0.1 * (rng.standard_normal((m.nR, m.dim, n, n)) + 1j * rng.standard_normal((m.nR, m.dim, n, n)))
    r[0] = 0.5 * (r[0] + r[0].conj().transpose(0, 2, 1))
    for i in range(1, m.nR, 2):  # R, -R follow each other
        r[i + 1] = r[i].conj().transpose(0, 2, 1)
    m.set_rmatrix(r)
    return m


@pytest.mark.parametrize("norb,rmat,nk", [(9, False, 3), (9, True, 70), (16, False, 5), (31, False, 200), (33, True, 3),
                                          (47, False, 2), (64, False, 40), (65, False, 2), (80, True, 2), (81, True, 2),
                                          (129, False, 3)])
def test_berry_matches_oracle(norb, rmat, nk):
    m = W.random_model(2, norb, False, 1, seed=300 + norb)
    if rmat:
        with_rmatrix(m, norb)
    k = np.random.default_rng(norb).uniform(0, 1, (nk, 2))
    p = Parameters.rank2((1, 1), [1.0, 0.3], [0.0, 1.0], [0.0])
    Om, E = m.berry_curvature_on(k, p)
    Omr, Er = O.berry_on(m, k, np.array([[1.0, 0.3], [0.0, 1.0]]))
    assert np.max(np.abs(E - Er)) <= 1e-10 * np.max(np.abs(Er))
    assert np.max(np.abs(Om - Omr)) <= 1e-8 * np.max(np.abs(Omr))
