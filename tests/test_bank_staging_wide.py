"""The seed-bank kernel's in-place conversion to one float4 per residue
(points_to_f4 in indialign_b200/csrc/k_bank.cu, launches of few items), replayed
on the CPU byte for byte beside the pair layout's in test_bank_staging: in round
r every thread of the 128-thread CTA first reads point 128r + tid, then (after a
barrier) writes {x, y, z, w}; the set is padded to a multiple of four points
that no cutoff selects.  Native points outside the mask become NaN."""
from __future__ import annotations

import numpy as np
import pytest

from test_bank_staging import CTA, _region_bytes


def _replay(points, lead, nmax, valid, native):
    n = points.shape[0]
    region = bytearray(_region_bytes(nmax))
    region[lead:lead + 24 * n] = points.astype("<f8").tobytes()
    off = points.mean(0)
    padded = (n + 3) & ~3
    for base in range(0, n, CTA):
        vals = {}
        for i in range(base, base + CTA):  # reads, before the barrier
            v = np.array([np.nan if native else 0.0, 0.0, 0.0, 1.0 if native else 0.0], "<f4")
            if i < n and (valid is None or valid[i] != 0 or not native):
                x = np.frombuffer(bytes(region[lead + 24 * i:lead + 24 * i + 24]), "<f8")
                v[:3] = (x - off).astype("<f4")
                v[3] = 1.0 if native or valid is None or valid[i] != 0 else 0.0
            vals[i] = v
        for i in range(base, base + CTA):  # writes, after it
            if i < padded:
                assert 16 * i + 16 <= lead + 24 * (base + CTA)  # below every later read
                assert 16 * i + 16 <= len(region)
                region[16 * i:16 * i + 16] = vals[i].tobytes()
    assert 16 * padded <= len(region)
    return np.frombuffer(bytes(region[:16 * padded]), "<f4").reshape(padded, 4)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 125, 126, 127, 128, 129, 130, 256, 257, 1000, 1501])
@pytest.mark.parametrize("lead", [0, 8])
def test_in_place_conversion_to_float4(n, lead):
    rng = np.random.default_rng(n + lead)
    pts = rng.standard_normal((n, 3)) * 30 + rng.uniform(-50, 50, 3)
    valid = (rng.uniform(size=n) > 0.2).astype(np.uint8) * rng.integers(1, 3, n).astype(np.uint8)
    want = (pts - pts.mean(0)).astype(np.float32)
    for v in (None, valid):
        on = np.ones(n, bool) if v is None else v != 0
        p = _replay(pts, lead, n, v, native=False)
        np.testing.assert_array_equal(p[:n, :3], want)
        np.testing.assert_array_equal(p[:n, 3], on.astype(np.float32))
        q = _replay(pts, lead, n, v, native=True)
        np.testing.assert_array_equal(q[:n, :3][on], want[on])
        assert np.isnan(q[:n, 0][~on]).all() and np.all(q[:, 3] == 1)
        # the padding: outside the mask on the pred side, NaN on the native side
        assert np.all(p[n:, 3] == 0) and np.isnan(q[n:, 0]).all()
