"""Seed-bank launches of few items (four lanes an item, csrc/k_bank.cu
wide_items) give the same bits as large launches (a thread an item): a pair
alone against the same pair inside a batch."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_alone_equals_in_a_batch():
    rng = np.random.default_rng(3)
    sizes = (3, 4, 5, 6, 31, 64, 66, 127, 257)  # every remainder of four residues, odd and even
    few = [W.make_pair(L, 4.0, rng, 0.1 if L > 6 else 0.0) for L in sizes]
    few[5].pred[7, 1] = np.inf  # a residue that no cutoff selects
    crowd = W.batch(160, 60, 120, seed=5)  # 160 x ~3000 items: beyond the line
    s, R, t = ia.search(few + crowd)
    for i, p in enumerate(few):
        s1, R1, t1 = ia.search([p])
        assert s1[0] == s[i] and np.array_equal(R1[0], R[i]) and np.array_equal(t1[0], t[i]), sizes[i]
