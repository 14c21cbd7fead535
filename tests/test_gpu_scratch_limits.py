"""Calls whose scratch does not fit take their smaller forms: sums and images in
parts, the direct Fourier sum, band tracking on the host (GPU).

Allocations beyond a limit set by the test fail as on a full device."""

import ctypes

import numpy as np
import pytest

from rustb_gb300 import _lib, workloads as W
from rustb_gb300.params import Integration, Parameters

pytestmark = pytest.mark.gpu


def limited(nbytes, f):
    """f() under the limit, and the kernel families that ran."""
    lib = _lib.load()
    cap = lib.tbg_internal_scratch_cap
    cap.restype, cap.argtypes = None, [ctypes.c_int64]
    lib.tbg_kernel_timing_enable(1)
    _lib.kernel_timing(reset=True)
    cap(nbytes)
    try:
        return f(), _lib.kernel_timing(reset=True)
    finally:
        cap(0)
        lib.tbg_kernel_timing_enable(0)


def test_fourier_sums_in_parts():
    m = W.random_model(2, 64, False, 1, seed=5)
    k = np.random.default_rng(5).uniform(0, 1, (300, 2))
    H = m.gen_ham_batch(k)
    # the sums' scratch is the size of H and a little more
    got, names = limited(H.nbytes + 32768, lambda: m.gen_ham_batch(k))
    assert names["oz64_fourier_kernel"][0] > 1
    assert np.array_equal(got, H)


def test_fourier_sums_without_scratch():
    m = W.random_model(3, 12, False, 4, seed=6)
    k = np.random.default_rng(6).uniform(0, 1, (300, 3))
    H, names = limited(0, lambda: m.gen_ham_batch(k))
    assert "oz64_fourier_kernel" in names
    # a row tile's image of the 365 pairs alone is 1.3 MB
    got, names = limited(1 << 20, lambda: m.gen_ham_batch(k))
    assert "oz64_fourier_kernel" not in names
    assert np.max(np.abs(got - H)) <= 1e-12 * np.max(np.abs(m.ham))


def test_no_room_for_the_tables_image():
    k = np.random.default_rng(9).uniform(0, 1, (200, 3))
    H, names = limited(0, lambda: W.random_model(3, 24, False, 2, seed=9).gen_ham_batch(k))
    assert "oz64_fourier_kernel" in names
    # 62 pairs of 576 columns take 2.1 MB, H 1.8 MB
    got, names = limited(2000000, lambda: W.random_model(3, 24, False, 2, seed=9).gen_ham_batch(k))
    assert "oz64_fourier_kernel" not in names
    assert np.max(np.abs(got - H)) <= 1e-12 * np.max(np.abs(H))


def test_product_images_in_parts():
    m = W.random_model(2, 40, False, 1, seed=7)
    k = np.random.default_rng(7).uniform(0, 1, (70, 2))
    p = Parameters.rank2((1, 1), [1.0, 0.0], [0.0, 1.0], [0.0])
    Om, E = m.berry_curvature_on(k, p)
    # V takes 3.6 MB, the images of its rows 12 MB
    (Omx, Ex), names = limited(6 << 20, lambda: m.berry_curvature_on(k, p))
    assert "oz64_kernel" in names
    assert np.array_equal(Omx, Om) and np.array_equal(Ex, E)


def test_energy_cut_overlaps(monkeypatch):
    m = W.random_model(3, 4, False, 1, seed=8)
    p = Parameters.rank2((12, 11, 10), [1.0, 0.0, 0.0], [0.0, 1.0, 0.0], list(np.linspace(-2, 2, 17)))
    p.eta = 0.05
    p.integration = Integration.EnergyCut
    monkeypatch.setenv("TBG_MAX_CHUNK", "64")
    ref, names = limited(0, lambda: m.hall_conductivity(p).conductivity)
    assert "ec_track_kernel" in names
    # vectors 338 KB, overlaps of the whole mesh 507 KB
    got, names = limited(400000, lambda: m.hall_conductivity(p).conductivity)
    assert "ec_track_kernel" not in names
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
