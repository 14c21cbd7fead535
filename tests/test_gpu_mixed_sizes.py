"""Mixed-precision Berry curvature and energies against the FP64 path (GPU) at
band counts around the tiles of the stages between them: 32 rows of the unpacked
Fourier sums, 64 columns and 128 rows of the float-pair products, odd lengths of
their FP32 and float-pair rows.

The path's own contract: energies to 1e-9 of the largest, curvature to 1e-6 of the
largest."""

import numpy as np
import pytest

from rustb_gb300 import workloads as W
from rustb_gb300.params import Parameters, Precision

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [31, 33, 64, 65, 96, 127, 129, 161])
def test_mixed_matches_fp64(nb):
    m = W.random_model(2, nb, False, 1, seed=nb)
    k = np.random.default_rng(nb).uniform(0, 1, (5, 2))
    p = Parameters.rank2((1, 1), np.array([1.0, 0.0]), np.array([0.0, 1.0]), [0.0])
    Om, E = m.berry_curvature_on(k, p, Precision.FP64)
    Omm, Em = m.berry_curvature_on(k, p, Precision.MIXED)
    assert np.abs(Em - E).max() < 1e-9 * max(1.0, np.abs(E).max())
    assert np.abs(Omm - Om).max() <= 1e-6 * np.abs(Om).max()
