"""Velocities of models whose on-site energies are far above the hoppings, and whose
hoppings fall steeply with |R|: the large sums are as accurate as the sum over R in
FP64 (GPU).

An FP64 sum of n terms is within n eps of the sum of their magnitudes; the bound here
is that with the largest |R| in it."""

import numpy as np
import pytest

from rustb_gb300 import workloads as W
from rustb_gb300.model import Model

pytestmark = pytest.mark.gpu


def reference(m, k):
    ph = np.exp(2j * np.pi * (k @ m.hamR.T)).astype(np.clongdouble)
    Rc = (m.hamR @ np.asarray(m.lat)).astype(np.longdouble)
    return [np.einsum("kr,rmn->kmn", 1j * ph * Rc[:, d], m.ham.astype(np.clongdouble)) for d in range(m.dim)]


@pytest.mark.parametrize("dim,n,rmax,decay", [(2, 24, 1, 0.0), (3, 20, 2, 0.0), (2, 14, 6, 2.0), (2, 30, 4, 4.0)])
def test_velocities(dim, n, rmax, decay):
    m = W.random_model(dim, n, False, rmax, seed=n)
    h = 0.01 * m.ham * np.exp(-decay * np.linalg.norm(m.hamR, axis=1))[:, None, None]
    h[0] += np.diag(np.linspace(-10.0, 10.0, n))
    m = Model(m.lat, m.orb, False, ham=h, hamR=m.hamR)
    k = np.random.default_rng(n).uniform(-1, 1, (400, dim))
    V, H = m.gen_v_batch(k, 0)
    terms = np.abs(h) * np.linalg.norm(m.hamR @ np.asarray(m.lat), axis=1)[:, None, None]
    for d, ref in enumerate(reference(m, k[:6])):
        err = np.abs(V[:6, d] - ref).max()
        assert err <= 4 * np.finfo(float).eps * terms.sum(0).max()
