"""Small models at the limits of their fused path: entries near the ends of FP64's
range, decoupled bands, k-points that are not finite (GPU)."""

import numpy as np
import pytest

from rustb_gb300 import Parameters
from rustb_gb300.model import Model

pytestmark = pytest.mark.gpu


def chain(onsite, hop):
    m = Model.tb_model(np.eye(2), [[0.0, 0.0], [0.5, 0.0]], spin=False)
    m.set_onsite(onsite)
    if hop:
        m.add_hop(hop, 0, 1, (0, 0))
    m.add_hop(0.0, 0, 0, (1, 0))
    return m


@pytest.mark.parametrize("onsite,hop", [([0.3, 1e-17], 0.0), ([1e200, -1e200], 1.0), ([1e-170, -3e-170], 0.0),
                                        ([-2e-320, 5e-310], 0.0), ([1e160, 1e160], 0.0), ([2.0, 1.0], 1e-18)])
def test_decoupled_bands_are_the_diagonal(onsite, hop):
    """The coupling is below the rounding of the diagonal: its entries are the energies."""
    E = chain(onsite, hop).solve_band_mesh((4, 3))
    assert np.array_equal(E, np.tile(np.sort(onsite), (12, 1)).reshape(E.shape))


def test_two_bands_match_the_closed_form():
    for d, h in [(1.0, 1.0), (1e-150, 1e-150), (1e150, 1e150), (1e-8, 1.0), (1.0, 1e-8), (0.0, 3.0)]:
        E = chain([d, -d], h).solve_band_mesh((3, 2)).reshape(-1, 2)
        r = np.hypot(d, h)
        assert np.max(np.abs(E - np.array([-r, r]))) <= 4 * np.finfo(float).eps * r


@pytest.mark.parametrize("k", [[0.1, np.nan], [0.1, np.inf], [np.nan, 0.2]])
def test_k_points_that_are_not_finite_give_no_numbers(k):
    """Also along an axis that no hopping uses."""
    m = chain([0.5, -0.5], 0.2)
    p = Parameters.rank2((1, 1), [1.0, 0.0], [0.0, 1.0], [0.0])
    Om, E = m.berry_curvature_on(np.array([k, [0.1, 0.2]]), p)
    assert not np.any(np.isfinite(E[0])) and not np.any(np.isfinite(Om[0]))
    assert np.all(np.isfinite(E[1])) and np.all(np.isfinite(Om[1]))
