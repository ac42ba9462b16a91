"""Undecided samples of an inverse transform, by how many a block has: none but the DC
(one evaluation for all 64), ties in 16, 32, 48 or all samples (the reference order by
columns), one to a few (fixed point, four at a time or one over the warp), and sums of
|coefficients| past what the fixed point takes. Every sample equals the oracle's."""
import ctypes

import numpy as np
import pytest

import oracle
from test_gpu_transform_stress import _first_mismatches, harness  # noqa: F401

pytestmark = pytest.mark.gpu

RATIONAL = [0, 4, 32, 36]  # (0,0), (0,4), (4,0), (4,4): weights +-1/8


def blocks(kind, n=40_000):
    rng = np.random.default_rng(7)
    c = np.zeros((n, 64), np.int32)
    if kind == "flat":
        c[:, 0] = rng.integers(-2100, 2100, n)
    elif kind == "flat_large":
        c[:, 0] = rng.integers(-2**31, 2**31, n)
    elif kind == "rational":
        c[:, RATIONAL] = rng.integers(-40, 41, (n, 4)) * (rng.random((n, 4)) < 0.8)
        c[:, 0] += rng.integers(-1000, 1000, n)
    elif kind == "rational_large":
        c[:, RATIONAL] = rng.integers(-40, 41, (n, 4)) << rng.integers(0, 22, (n, 1))
    elif kind == "one_column":  # ties where the odd terms cancel or vanish
        c[:, RATIONAL] = rng.integers(-8, 9, (n, 4))
        c[np.arange(n), rng.integers(0, 64, n)] += rng.integers(-3, 4, n)
    else:  # a few undecided samples a block: a wide fp32 bound
        c[:] = rng.integers(-2**14, 2**14, (n, 64)) * (rng.random((n, 64)) < 0.6)
    return c


@pytest.mark.parametrize("kind", ["flat", "flat_large", "rational", "rational_large", "one_column", "wide"])
def test_settled_samples_equal_the_oracle(harness, kind):  # noqa: F811
    c = blocks(kind)
    gpu = np.empty((len(c), 64), np.uint8)
    exact = ctypes.c_ulonglong(0)
    assert harness.harness_jpeg_idct(c.ctypes.data, len(c), gpu.ctypes.data, ctypes.byref(exact)) == 0
    bad, msg = _first_mismatches(gpu, oracle.jpeg_idct_many(c), kind, c)
    assert len(bad) == 0, msg
    assert exact.value > 0 or kind == "flat_large"  # (all clamped)
