"""What calls borrow and give back: models made and dropped one after the other, and
many at once, leave no device memory behind (GPU)."""

import concurrent.futures as cf

import numpy as np
import pytest
import torch

from rustb_gb300 import Parameters, workloads as W

pytestmark = pytest.mark.gpu


def one(i):
    m = W.haldane_200(t2=0.1 + 0.001 * i)
    s = m.hall_conductivity(Parameters.rank2((11, 11), [1.0, 0.0], [0.0, 1.0], [0.0])).conductivity
    m._invalidate()
    return s


def test_models_one_after_the_other_and_many_at_once():
    ref = [one(i) for i in range(12)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        assert all(np.array_equal(one(i), ref[i]) for i in range(12))
        with cf.ThreadPoolExecutor(12) as ex:
            assert all(np.array_equal(a, b) for a, b in zip(ex.map(one, range(12)), ref))
    torch.cuda.synchronize()
    # one lane (1.1 MB) stays; the driver hands out 2 MB at a time
    assert free - torch.cuda.mem_get_info()[0] <= 4 << 20
