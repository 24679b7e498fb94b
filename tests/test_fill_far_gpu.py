"""The distance fill on non-finite points and on points whose squared distances
leave the FP32 range: a NaN or infinite distance scores 0 and ends no path, and
far points that coincide score like near ones."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from test_nw_fill import _path

pytestmark = pytest.mark.gpu

FAR = float(2 ** 62)  # 4.6e18; differences of such points square beyond FP32


def _points(n, rng, kind):
    """Points on a coarse grid, some of them replaced."""
    P = rng.integers(-12, 13, (n, 3)) / 2.0
    at = rng.permutation(n)[:max(1, n // 3)]
    if kind == "nonfinite":
        P[at, rng.integers(0, 3, len(at))] = rng.choice([np.nan, np.inf, -np.inf], len(at))
    elif kind == "far":
        P[at, 2] = rng.choice([FAR, -FAR, 4 * FAR, 1e30, -1e37, 1e39], len(at))
    elif kind == "limit":  # the limit itself, and where the fill puts what lies beyond it
        P[at] = rng.choice([1e18, 2e18], len(at))[:, None] * rng.choice([-1, 1], (len(at), 3))
    return P


@pytest.mark.parametrize("warps", [1, 4])
@pytest.mark.parametrize("pkind,qkind", [("nonfinite", "nonfinite"), ("far", "far"), ("far", "near"), ("near", "far"),
                                         ("limit", "limit"), ("nonfinite", "far"), ("limit", "near")])
@pytest.mark.parametrize("plen,nlen", [(3, 4), (40, 31), (130, 97), (385, 70)])
def test_fill_of_far_and_non_finite_points(plen, nlen, pkind, qkind, warps):
    import indialign_b200 as ia
    rng = np.random.default_rng(plen * 7 + nlen + len(pkind))
    P, Q = _points(plen, rng, pkind), _points(nlen, rng, qkind)
    rt = np.array([0, 1, 0, -1, 0, 0, 0, 0, 1, 1.5, -2, 0], np.float64)
    with np.errstate(all="ignore"):
        # the permutation spelled out: 0 times infinity is NaN, as in the kernel's sums
        R = rt[:9].reshape(3, 3)
        moved = (P[:, :1] * R[0] + P[:, 1:2] * R[1] + P[:, 2:] * R[2] + rt[9:]).astype(np.float32)
        d = moved[:, None] - Q.astype(np.float32)[None]
        d2 = d[..., 2] * d[..., 2] + (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1])
        r = np.float32(1) / (np.float32(1) + d2 * np.float32(0.125))
        M = np.where(d2 <= np.float32(90), r, np.float32(0))
    assert np.isfinite(M).all()
    if (pkind, qkind) == ("far", "far") and plen > 3:
        assert M[np.abs(moved[:, 2]) > 1e18].any()  # far points that coincide
    f = ia.load().indialign_selftest_nw
    f.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] * 5 + [ctypes.c_int] + [ctypes.c_float] * 3 + [ctypes.c_int] + [ctypes.c_void_p] * 3
    lab = np.full(max(plen, nlen), ord("L"), np.uint8)
    for gap in (0.0, np.float32(-0.6)):
        ap, an, na = np.zeros(min(plen, nlen), np.int32), np.zeros(min(plen, nlen), np.int32), np.zeros(1, np.int32)
        assert f(plen, nlen, P.ctypes.data, Q.ctypes.data, rt.ctypes.data, lab.ctypes.data, lab.ctypes.data, 0, gap,
                 0.125, 90.0, warps, ap.ctypes.data, an.ctypes.data, na.ctypes.data) == 0
        assert list(zip(ap[:na[0]], an[:na[0]])) == _path(M, gap), gap


@pytest.mark.parametrize("n", [2, 40])  # a chain per CTA, a chain per warp
def test_far_pair_leaves_the_others_alone(n):
    """A batch with a far pair takes the far kernels for all of it: the other
    pairs' results are the same bits."""
    import indialign_b200 as ia
    from indialign_b200 import workloads as W
    pairs = W.batch(n, 40, 120, seed=31, sigma_lo=4.0, sigma_hi=14.0)
    far = W.Pair(pairs[0].pred + 1e19, pairs[0].native + 1e19,
                 *(getattr(pairs[0], k) for k in ("valid", "pred_valid", "native_valid", "lnorm")))
    s, R, t = ia.search(pairs)
    s2, R2, t2 = ia.search([far] + pairs[1:])
    assert np.isfinite(s2).all()
    for a, b in ((s, s2), (R, R2), (t, t2)):
        assert np.array_equal(a[1:], b[1:])
