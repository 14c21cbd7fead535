"""The centred form of the DOS kernel at the sizes where its runs, tiles and
windows change, against the closed sum in numpy over the GPU's own energies (GPU).

A term loses at most about 64 multiplications (64 eps) from the run and A^2 eps from
its arguments, where A^2 exp(-A^2 / 2) < 1; the bound is 1e-13 of the largest value."""

import numpy as np
import pytest

import models as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npt,sigma", [(2, 3.0), (255, 0.05), (256, 0.01), (257, 0.02), (500, 0.01), (513, 0.5),
                                       (600, 0.05), (600, 0.15), (64, 0.03), (37, 0.06)])
def test_dos_matches_the_sum(npt, sigma):
    m = M.haldane()
    E, d = m.dos([23, 19], -4.0, 4.0, npt, sigma)
    e = m.solve_band_mesh([23, 19]).reshape(-1)
    ref = np.exp(-(((E[:, None] - e[None, :]) / sigma) ** 2) / 2.0).sum(1) / (sigma * np.sqrt(2.0 * np.pi) * 23 * 19)
    assert np.max(np.abs(d - ref)) <= 1e-13 * np.max(ref)
