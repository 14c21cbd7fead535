"""A bounded wait that runs out in the FP64 digit products, in each form of a
contraction: reported as such, and the next product is right (GPU)."""

import numpy as np
import pytest

from rustb_gb300 import _lib, errors
from test_gpu_oz64 import case, gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 128, 200, 300])
def test_timeout_is_reported_and_recovers(K):
    A, B, ref, scale = case(4, 130, 70, K, 0, 0, K)
    lib = _lib.load()
    prev = lib.tbg_internal_tc_wait_limit(1)
    try:
        with pytest.raises(errors.DeviceError) as ei:
            gemm(A, B, np.zeros_like(ref, dtype=complex), 0, 0, 0)
        assert ei.value.code == errors.TBG_E_TIMEOUT
    finally:
        lib.tbg_internal_tc_wait_limit(prev)
    got = gemm(A, B, np.zeros_like(ref, dtype=complex), 0, 0, 0)
    assert np.all(np.abs(got - ref) <= 16.0 * (K + 8) * 2.0 ** -54 * scale)
