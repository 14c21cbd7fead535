"""Host threads solving FP64 models of different sizes at once: the reduction of
the larger ones launches with a shared-memory footprint of its own per size (GPU)."""

import concurrent.futures as cf

import numpy as np
import pytest

from rustb_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_concurrent_calls_on_large_models():
    sizes = [(170, 24), (200, 24), (300, 12), (512, 6)]
    models = [W.random_model(2, n, False, 1, seed=900 + n) for n, _ in sizes]
    ks = [np.random.default_rng(n).uniform(0, 1, (nk, 2)) for n, nk in sizes]
    alone = [m.solve_band_all_parallel(k) for m, k in zip(models, ks)]

    def run(i):
        return [models[i].solve_band_all_parallel(ks[i]) for _ in range(6)]

    with cf.ThreadPoolExecutor(len(models)) as ex:
        out = list(ex.map(run, range(len(models))))
    for a, rs in zip(alone, out):
        for r in rs:
            assert np.array_equal(a, r)
