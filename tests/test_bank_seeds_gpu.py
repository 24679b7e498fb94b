"""The seeds' own Kabsch (csrc/k_bank.cu k_bank_seeds) at its edges: one and
several blocks of 128 seeds, windows shorter and longer than the unrolled loop,
anchor bitmasks, mask bytes other than 0 and 1 (windows take nonzero bytes,
bitmasks 1 & byte), and a point set too large for shared memory."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import abi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,values", [(4, (1,)), (5, (0, 1, 1)), (31, (0, 1, 2, 3)), (67, (1, 2)), (130, (0, 1, 1, 255)),
                                      (260, (0, 1, 3, 5))])
def test_seed_bank_best_matches_the_oracle(oracle, L, values):
    rng = np.random.default_rng(L)
    p = W.make_pair(L, 3.0, rng)
    p.valid = rng.choice(values, L).astype(np.uint8)
    p.pred_valid = p.native_valid = p.valid
    best = np.zeros(ia.TRACE_STAGES * 13)
    s, R, t = ia.search([p], stage_best=best)
    rc, so, _, _ = abi.run_batch(oracle, [p], prefix="ora_")
    assert rc == 0 and s[0] >= so[0] - 1e-6
    if so[0] == 0.0:  # no seed with three valid residues: score 0, identity
        assert s[0] == 0.0
        return
    # the recorded bank best is the score of its own transform
    m = p.pred @ best[1:10].reshape(3, 3) + best[10:13]
    d0 = max(0.6 * np.sqrt(L - 0.5) - 2.5, 0.3) if L >= 30 else [0.3, 0.4, 0.5, 0.6, 0.7][sum(L > k for k in (11, 15, 19, 23))]
    tm = (1 / (1 + ((m - p.native) ** 2).sum(1) / d0 ** 2))[p.valid != 0].sum() / p.lnorm
    assert best[0] == pytest.approx(tm, abs=1e-9)


def test_global_path_equals_the_shared_one():
    """6800 residues do not fit k_bank_seeds' shared memory and 12100 not
    k_anchor's, 6000 fit both: the same chain, invalid beyond 900 residues,
    scores the same on every path."""
    rng = np.random.default_rng(9)
    base = W.make_pair(900, 2.0, rng)
    out = []
    for N in (6000, 6800, 12100):
        pad = lambda a: np.concatenate([a, np.zeros((N - 900,) + a.shape[1:], a.dtype)])  # noqa: E731
        p = W.Pair(pad(base.pred), pad(base.native), *(pad(base.valid) for _ in range(3)), 900.0)
        out.append(ia.search([p])[0][0])
    assert out[1:] == pytest.approx([out[0]] * 2, abs=1e-6)
