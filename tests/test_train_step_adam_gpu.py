"""The training step's weight update (k_step_finish) against Adam in FP64 from
the step's own gradient and the moments before it, and its gradients against the
single calls' with a bound that narrows with the batch."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import ranker

pytestmark = pytest.mark.gpu

U = 2.0 ** -24  # half an ulp of FP32, relative


def _data(n):
    import torch
    rng = np.random.default_rng(n + 5)
    x = rng.normal(0.3, 1.7, (n, ia.FEATURES)).astype(np.float32)
    t = rng.uniform(0, 1, n).astype(np.float32)
    blob = ranker.init_blob(np.full(ia.FEATURES, 0.3, np.float32), np.full(ia.FEATURES, 1.7, np.float32), n)
    return torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda"), blob


@pytest.mark.parametrize("n", [1, 64, 1003])
@pytest.mark.parametrize("lr,beta1,beta2,eps", [(1e-3, 0.9, 0.999, 1e-8), (3e-2, 0.5, 0.9, 1e-4)])
def test_weights_follow_adam(n, lr, beta1, beta2, eps):
    X, T, blob = _data(n)
    tr = ranker.Trainer(blob, batch=n, lr=lr, lam=0.7, beta1=beta1, beta2=beta2, eps=eps)
    f64 = lambda a: a.double().cpu().numpy()  # noqa: E731
    b1, b2, rate, e = (float(np.float32(k)) for k in (beta1, beta2, lr, eps))
    c1, c2 = float(np.float32(1) - np.float32(b1)), float(np.float32(1) - np.float32(b2))
    for step in (1, 2, 3):
        w0, m0, v0 = f64(tr.blob), f64(tr.m), f64(tr.v)
        tr.step(X, T)
        g, w, m, v = f64(tr.grad), f64(tr.blob), f64(tr.m), f64(tr.v)
        head = slice(0, ranker.W1)  # mean and deviation of the features are not trained
        assert not g[head].any() and np.array_equal(w[head], w0[head])
        assert g[ranker.W1:].any()
        # two products and a sum, each rounded once; denormal squares to their last bit
        assert np.all(np.abs(m - (b1 * m0 + c1 * g)) <= 3 * U * (np.abs(b1 * m0) + np.abs(c1 * g)) + 2.0 ** -148)
        assert np.all(np.abs(v - (b2 * v0 + c2 * g * g)) <= 4 * U * (b2 * v0 + c2 * g * g) + 2.0 ** -147)
        # the update from the stored moments: eight rounded operations, then the subtraction's rounding
        bc1, bc2 = (float(np.float32(1 - b ** step)) for b in (b1, b2))
        u = rate * (m / bc1) / (np.sqrt(v / bc2) + e)
        t = slice(ranker.W1, None)
        assert np.all(np.abs(w - (w0 - u))[t] <= (8 * U * np.abs(u) + U * np.abs(w0 - u) + 2.0 ** -148)[t])
        assert np.abs(w - w0)[t].max() > 0.1 * rate


@pytest.mark.parametrize("n", [129, 1003, 8192])
def test_gradients_of_larger_batches_agree_closely(n):
    """As the single calls' up to the order of FP32 sums and to turned BF16
    roundings of dz1, dz2: a relative difference of 1e-6 turns one in 4000 of
    them, by 2^-8 of the value, so a block's norm moves by 2^-8 / 64 or, where
    that is less than one entry, by 2^-8 / sqrt(128 n); four times that."""
    X, T, blob = _data(n)
    a, b = (ranker.Trainer(blob, batch=n, lam=0.7) for _ in range(2))
    a.gradients(X, T)
    b.step(X, T)
    rel = 4 * 2.0 ** -8 * max(2.0 ** -6, (128 * n) ** -0.5)
    edges = (ranker.W1, ranker.B1, ranker.W2, ranker.B2, ranker.W3, ranker.B3, ranker.B3 + 1)
    for lo, hi in zip(edges, edges[1:]):
        d = (b.grad[lo:hi].double() - a.grad[lo:hi].double()).norm()
        assert d <= rel * a.grad[lo:hi].double().norm() + 1e-9, lo
