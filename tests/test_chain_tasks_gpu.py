"""Chain launches of every size (csrc/k_chain.cu: a CTA per chain, a few chains
per CTA, many chains per warp) give a pair the same bits: alone, and in batches
whose launches have from tens to hundreds of thousands of chains."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def alone():
    rng = np.random.default_rng(17)
    pairs = [W.make_pair(L, 9.0, rng, 0.15 if L > 6 else 0.0) for L in (3, 5, 40, 97, 128, 129, 260)]
    return pairs, [ia.search([p]) for p in pairs]


@pytest.mark.parametrize("crowd", [0, 1, 25, 200])
def test_batch_equals_alone(alone, crowd):
    pairs, one = alone
    rest = W.batch(crowd, 30, 200, seed=9) if crowd else []
    s, R, t = ia.search(pairs + rest)
    for i, (s1, R1, t1) in enumerate(one):
        assert s1[0] == s[i] and np.array_equal(R1[0], R[i]) and np.array_equal(t1[0], t[i]), i
