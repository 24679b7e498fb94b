"""The kernels' FP64 reciprocal and quotient (rcp_cr, div_by) against the
division: equal, save the reciprocal of a mantissa of all ones, which may be an
ulp off."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _division(a, b):
    import indialign_b200 as ia
    f = ia.load().indialign_selftest_division
    f.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4
    y, q = np.zeros_like(a), np.zeros_like(a)
    assert f(len(a), a.ctypes.data, b.ctypes.data, y.ctypes.data, q.ctypes.data) == 0
    return y, q


def _mantissas(rng, n):
    """1 <= m < 2: random ones, and those at either end of the range."""
    bits = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    bits[::16] = rng.integers(0, 64, len(bits[::16]), dtype=np.uint64)
    bits[1::16] = (1 << 52) - 1 - rng.integers(0, 64, len(bits[1::16]), dtype=np.uint64)
    return (bits | np.uint64(0x3FF << 52)).view(np.float64)


@pytest.mark.parametrize("kind", ["counts", "weights", "terms"])
def test_reciprocal_and_quotient(kind):
    """Point counts, weight sums and TM terms 1 + d2 / d0^2, under sums of any sign and size."""
    rng = np.random.default_rng(len(kind))
    n = 1 << 21
    if kind == "counts":
        b = rng.integers(3, 65536, n).astype(np.float64)
    elif kind == "weights":
        b = _mantissas(rng, n) * 2.0 ** rng.integers(-40, 17, n)
    else:
        b = _mantissas(rng, n) * 2.0 ** rng.integers(0, 900, n)
    a = _mantissas(rng, n) * rng.choice([-1.0, 1.0], n) * 2.0 ** rng.integers(-30, 60, n)
    y, q = _division(a, b)
    ones = (b.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)
    assert np.array_equal(y[~ones], (1.0 / b)[~ones])
    assert np.all(np.abs(y - 1.0 / b)[ones] <= np.spacing(1.0 / b)[ones])
    if kind != "terms":
        assert np.array_equal(q[~ones], (a / b)[~ones])
        assert np.all(np.abs(q - a / b)[ones] <= np.spacing(np.abs(a / b))[ones])


def test_ends_of_the_range():
    b = np.array([1.0, 2.0 ** 1021, 2.0 ** 1023, np.inf, np.nan])
    y, _ = _division(np.ones_like(b), b)
    assert y[0] == 1.0 and y[1] == 2.0 ** -1021 and 0.0 <= y[2] <= 2.0 ** -1022
    assert np.isnan(y[4])
