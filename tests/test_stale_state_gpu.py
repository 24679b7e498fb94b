"""A search does not depend on what an earlier batch left in the device state:
pairs without a finite score first, then ordinary ones in the same places."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import ranker, workloads as W

pytestmark = pytest.mark.gpu


def test_learned_search_after_pairs_without_a_score():
    rng = np.random.default_rng(71)
    pairs = [W.make_pair(L, float(rng.uniform(0.5, 14)), rng, 0.05) for L in (40, 128, 200, 300)]
    broken = [W.make_pair(L, 4.0, rng) for L in (64, 64, 64, 64)]
    for p in broken:
        p.pred[7, 1] = np.inf
    blob, out = ranker.default_weights(), []
    for first in (pairs, broken):
        ia.search(first, ranker=blob)
        ct, st = np.zeros(ia.COUNTERS, np.int64), np.zeros(ia.RANK_STATS, np.int64)
        s, R, t = ia.search(pairs, ranker=blob, counters=ct, rank_stats=st)
        out.append((s, R, t, ct[0], st))  # ct[0]: cells of the alignments
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
