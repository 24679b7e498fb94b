"""Launches are planned by one CTA up to 512 tasks (one task per pair, or two)
and by a grid beyond: batches on both sides of each line give every pair the
bits that it has in a small batch."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    pairs = W.batch(513, 20, 48, seed=23)
    parts = [ia.search(pairs[i:i + 27]) for i in range(0, 513, 27)]
    return pairs, [np.concatenate([p[k] for p in parts]) for k in range(3)]


@pytest.mark.parametrize("n", [1, 33, 256, 257, 512, 513])
def test_batch_equals_small_batches(small, n):
    pairs, want = small
    for got, w in zip(ia.search(pairs[:n]), want):
        np.testing.assert_array_equal(got, w[:n])
