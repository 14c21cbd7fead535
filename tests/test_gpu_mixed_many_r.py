"""MIXED curvature of models with more R vectors than the float-pair contraction
takes: the FP64 sums behind it run on the tensor cores as they do in FP64 (GPU)."""

import numpy as np
import pytest

from rustb_gb300 import Parameters, _lib, workloads as W
from rustb_gb300.params import Precision

pytestmark = pytest.mark.gpu


def test_many_hoppings():
    m = W.random_model(3, 40, False, 4, seed=77)  # 729 R
    k = np.random.default_rng(4).uniform(0, 1, (200, 3))
    p = Parameters.rank2((1, 1, 1), [1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0])
    Om, E = m.berry_curvature_on(k, p)
    lib = _lib.load()
    lib.tbg_kernel_timing_enable(1)
    _lib.kernel_timing(reset=True)
    Omx, Ex = m.berry_curvature_on(k, p, Precision.MIXED)
    names = _lib.kernel_timing(reset=True)
    lib.tbg_kernel_timing_enable(0)
    assert "oz64_fourier_kernel" in names and "fourier_gemm_kernel" not in names
    # the mixed path's bounds: energies 1e-9 ||H||, curvature 1e-6 of its largest value
    assert np.max(np.abs(Ex - E)) <= 1e-9 * np.max(np.abs(E))
    assert np.max(np.abs(Omx - Om)) <= 1e-6 * np.max(np.abs(Om))
