"""Band tracking of the energy-cut integration on the GPU and on the host: the same
result wherever both can run, and the host's against the oracle above the GPU's band
count (GPU)."""

import ctypes

import numpy as np
import pytest

from oracle import tb_oracle as O
from rustb_gb300 import _lib, workloads as W
from rustb_gb300.params import Integration, Parameters

pytestmark = pytest.mark.gpu
MU = np.linspace(-2.0, 2.0, 17)


def ec(m, kmesh):
    p = Parameters.rank2(kmesh, np.eye(m.dim)[0], np.eye(m.dim)[1], list(MU))
    p.eta = 0.05
    p.integration = Integration.EnergyCut
    return m.hall_conductivity(p).conductivity


def kernels(f):
    lib = _lib.load()
    lib.tbg_kernel_timing_enable(1)
    _lib.kernel_timing(reset=True)
    r = f()
    names = _lib.kernel_timing(reset=True)
    lib.tbg_kernel_timing_enable(0)
    return r, names


@pytest.mark.parametrize("n", [1, 2, 3, 4])
@pytest.mark.parametrize("kmesh", [(40, 33), (33, 40), (1, 9), (12, 11, 10)])
def test_gpu_and_host_agree(n, kmesh):
    lib = _lib.load()
    hook = lib.tbg_internal_ec_track_max
    hook.restype, hook.argtypes = ctypes.c_int, [ctypes.c_int]
    m = W.random_model(len(kmesh), n, False, 1, seed=60 + n)
    got, names = kernels(lambda: ec(m, kmesh))
    assert "ec_track_kernel" in names
    hook(0)
    try:
        ref, names = kernels(lambda: ec(m, kmesh))
    finally:
        hook(-1)
    assert "ec_track_kernel" not in names
    # the same permutations: only the order of the integration's atomic sums differs
    assert np.max(np.abs(got - ref)) <= 1e-12 * max(np.max(np.abs(ref)), 1e-3)


@pytest.mark.parametrize("n,kmesh", [(4, (3, 300)), (4, (24, 24, 2)), (9, (9, 8)), (12, (5, 6)), (10, (4, 3, 3))])
def test_host_tracking_matches_oracle(n, kmesh):
    """Long and flat meshes, and more bands than the GPU tracks."""
    m = W.random_model(len(kmesh), n, False, 1, seed=80 + n)
    got, names = kernels(lambda: ec(m, kmesh))
    assert "ec_track_kernel" not in names
    ref = O.hall_energy_cut(m, list(kmesh), np.eye(len(kmesh))[:2], MU, 0.0, 0.05)
    assert np.max(np.abs(got - ref)) <= 1e-9 * max(np.max(np.abs(ref)), 1e-3)
