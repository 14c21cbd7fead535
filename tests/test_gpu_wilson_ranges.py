"""Wannier centres of bands that do not start at the lowest, of sets with gaps and of
several loops, at the sizes where only part of the vectors is made and where the
overlaps run on the tensor cores; phases against the oracle (GPU)."""

import numpy as np
import pytest

from oracle import tb_oracle as O
from rustb_gb300 import workloads as W
from test_gpu_wilson import same_phases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,occ", [(20, [5, 6, 7, 8]), (33, list(range(12))), (33, list(range(7, 21))),
                                   (33, list(range(21, 33))), (40, list(range(0, 30, 2))), (40, [31, 4, 17]),
                                   (64, list(range(16, 48))), (64, list(range(1, 64))), (97, list(range(30, 60)))])
def test_wannier_centres(n, occ):
    m = W.random_model(2, n, False, 1, seed=900 + n)
    args = (occ, np.array([0.05, 0.0]), np.array([1.0, 0.0]), np.array([0.0, 1.0]), 5, 21)
    got, ref = m.wannier_centre(*args), O.wannier_centre(m, *args)
    for c in range(5):
        assert same_phases(got[:, c], ref[:, c])
