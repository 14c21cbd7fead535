"""A call on the same model and k-points gives the same bits every time (GPU)."""

import numpy as np
import pytest

from rustb_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(16, 64), (64, 40), (128, 20), (170, 12), (300, 6), (512, 3)])
def test_bands_are_the_same_every_time(n, nk):
    m = W.random_model(2, n, False, 1, seed=n)
    k = np.random.default_rng(n).uniform(0, 1, (nk, 2))
    first = m.solve_band_all_parallel(k)
    for _ in range(4):
        assert np.array_equal(first, m.solve_band_all_parallel(k))
