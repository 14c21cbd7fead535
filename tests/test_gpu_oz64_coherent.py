"""FP64-accurate tensor-core products of operands whose digits are large and whose
terms all add up, the largest sums an accumulator can meet (GPU).

Zero-mean operands leave the digit sums two orders of magnitude below FP32's 24
bits; these reach them.  The bound is that of test_gpu_oz64."""

import numpy as np
import pytest

from rustb_gb300 import workloads as W
from test_gpu_oz64 import gemm

pytestmark = pytest.mark.gpu

# with |x| < 2^E a value is written on the grid 2^(E - 55) as digits of eight bits
TOP = 254.0 / 255.0   # every digit 127
MID = 14.0 / 17.0     # every digit 105


def values(rng, shape, kind):
    if kind == "digits":  # all digits in 112 .. 127
        x = np.zeros(shape)
        for s in range(7):
            x = x * 256.0 + rng.integers(112, 128, shape)
        return x * 2.0 ** -55
    base, spread = kind
    return base * (1.0 - spread * rng.uniform(0, 1, shape))


KINDS = ["digits", (TOP, 0.0), (TOP, 3e-12), (TOP, 3e-10), (TOP, 1e-7), (MID, 0.0), (MID, 3e-12), (MID, 3e-10),
         (MID, 1e-7)]


@pytest.mark.parametrize("K", [16, 64, 96, 97, 103, 127, 128, 129, 144, 172, 192, 200, 256, 257, 300, 384, 600])
def test_coherent_products(K):
    """Re and Im of A and of conj(B) positive: all 2 K terms of a real part add."""
    rng = np.random.default_rng(K)
    for kind in KINDS:
        A = values(rng, (1, 40, K), kind) + 1j * values(rng, (1, 40, K), kind)
        B = values(rng, (1, K, 33), kind) - 1j * values(rng, (1, K, 33), kind)
        ref = np.einsum("bmk,bkn->bmn", A.astype(np.clongdouble), B.astype(np.clongdouble))
        scale = np.abs(A).max(2)[:, :, None] * np.abs(B).max(1)[:, None, :]
        got = gemm(A, B, np.zeros(ref.shape, complex), 0, 0, 0)
        assert np.all(np.abs(got - ref) <= 16.0 * (K + 8) * 2.0 ** -54 * scale), kind
        C0 = np.ones(ref.shape, complex)
        sub = gemm(A, B, C0, 0, 0, -1)
        assert np.all(np.abs(sub - (C0 - ref)) <= 32.0 * (K + 8) * 2.0 ** -54 * scale), kind


@pytest.mark.parametrize("K", [128, 256])
def test_negative_digits(K):
    """The most negative digits (-128 below the first) and both signs of the sum."""
    rng = np.random.default_rng(K + 1)
    x = (127.0 - 128.0 * sum(256.0 ** -s for s in range(1, 7))) / 128.0  # digit 0 is 127, the others -128
    for sign in (1.0, -1.0):
        A = x * (1.0 - 2.0 ** -50 * rng.integers(0, 2, (1, 40, K))) * (1 + 1j)
        B = sign * x * (1.0 - 2.0 ** -50 * rng.integers(0, 2, (1, K, 32))) * (1 - 1j)
        ref = np.einsum("bmk,bkn->bmn", A.astype(np.clongdouble), B.astype(np.clongdouble))
        scale = np.abs(A).max(2)[:, :, None] * np.abs(B).max(1)[:, None, :]
        got = gemm(A, B, np.zeros(ref.shape, complex), 0, 0, 0)
        assert np.all(np.abs(got - ref) <= 16.0 * (K + 8) * 2.0 ** -54 * scale)


@pytest.mark.parametrize("rmax,n", [(3, 24), (4, 20), (5, 16)])
def test_fourier_sums_of_many_pairs(rmax, n):
    """Table products of 172, 365 and 666 pairs against the sum over R."""
    m = W.random_model(3, n, False, rmax, seed=40 + rmax)
    k = np.random.default_rng(rmax).uniform(-1, 1, (400, 3))
    H = m.gen_ham_batch(k, 0)
    ph = np.exp(2j * np.pi * (k @ m.hamR.T))
    ref = np.einsum("kr,rmn->kmn", ph, m.ham)
    assert np.max(np.abs(H - ref)) <= 64 * m.nR * 2.0 ** -53 * np.max(np.abs(m.ham))
