"""Pairs with valid residues whose native (or pred) mask is empty, first, in the
middle and last in the batch: they have seeds, and chains over a side without
residues.  The GPU library against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from indialign_b200 import abi, workloads as W


def _pair(N, rng, pv, nv):
    x = W.make_trace(N, rng)
    nat = (x + rng.normal(0, 2.0, (N, 3))) @ W.random_rotation(rng).T + rng.uniform(-20, 20, 3)
    return W.Pair(np.ascontiguousarray(x), np.ascontiguousarray(nat), np.ones(N, np.uint8), pv.astype(np.uint8),
                  nv.astype(np.uint8), float(N))


def _cases():
    rng = np.random.default_rng(5)
    out = []
    for N in (12, 40, 67):
        one, zero = np.ones(N, bool), np.zeros(N, bool)
        two = np.arange(N) < 2
        out += [_pair(N, rng, one, zero), _pair(N, rng, one, one), _pair(N, rng, zero, one),
                _pair(N, rng, zero, zero), _pair(N, rng, one, two), _pair(N, rng, two, one), _pair(N, rng, one, zero)]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("alone", [True, False])
def test_empty_sides_gpu_vs_oracle(oracle, alone):
    import indialign_b200 as ia
    pairs = _cases()
    rc, so, _, _ = abi.run_batch(oracle, pairs, prefix="ora_")
    assert rc == 0
    s = np.concatenate([ia.search([p])[0] for p in pairs]) if alone else ia.search(pairs)[0]
    assert np.all(s >= so - 1e-6) and np.all(s <= 1.0 + 1e-9), (s, so)
