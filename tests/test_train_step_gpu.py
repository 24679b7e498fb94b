"""The one-call training step (indialign_mlp_step) against the same step by its
single calls (forward, loss, backward, Adam, pack), at the edges of its row
tiles (16 rows a warp, 64 a CTA, 128 a tensor-core tile) and of the split-K."""
from __future__ import annotations

import numpy as np
import pytest

import indialign_b200 as ia
from indialign_b200 import ranker

pytestmark = pytest.mark.gpu

# Both run the same products on the same BF16 operands and add in another FP32
# order (1e-6 of a block's norm); a difference in the last bit of a value may
# turn one BF16 rounding of dz1, which is 2^-8 of one of a row's 128 entries.
REL = 2.0 ** -8 / 128 ** 0.5 * 4


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 128, 129, 500, 1003, 8192])
def test_step_equals_its_parts(n):
    import ctypes
    import torch
    rng = np.random.default_rng(n)
    x = rng.normal(0.3, 1.7, (n, ia.FEATURES)).astype(np.float32)
    t = rng.uniform(0, 1, n).astype(np.float32)
    t[1::7] = t[0:n - 1:7][:len(t[1::7])]  # ties: pairs without a ranking term
    blob = ranker.init_blob(np.full(ia.FEATURES, 0.3, np.float32), np.full(ia.FEATURES, 1.7, np.float32), n)
    X, T = torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda")
    a, b = (ranker.Trainer(blob, batch=max(n, 40), lam=0.7) for _ in range(2))
    for step in (1, 2):
        for dst, src in ((a.blob, b.blob), (a.m, b.m), (a.v, b.v)):
            dst.copy_(src)
        a.pack()
        la, ga = a.gradients(X, T)
        la, ga, ya = float(la.item()), ga.double().clone(), a.y[:n].clone()
        f = ctypes.c_float
        assert a.lib.indialign_mlp_adam(a.blob.data_ptr(), a.grad.data_ptr(), a.m.data_ptr(), a.v.data_ptr(), step,
                                        f(a.lr), f(a.beta1), f(a.beta2), f(a.eps), a.stream) == 0
        lb = float(b.step(X, T).item())
        assert torch.equal(ya, b.y[:n])
        assert lb == pytest.approx(la, rel=1e-5)
        for lo, hi in ((0, ranker.W1), (ranker.W1, ranker.B1), (ranker.B1, ranker.W2), (ranker.W2, ranker.B2),
                       (ranker.B2, ranker.W3), (ranker.W3, ranker.B3), (ranker.B3, ranker.B3 + 1)):
            d = (b.grad[lo:hi].double() - ga[lo:hi]).norm()
            assert d <= REL * ga[lo:hi].norm() + 1e-9, (step, lo)
        assert (a.m - b.m).norm() <= REL * a.m.norm() and (a.v - b.v).norm() <= 2 * REL * a.v.norm()
        assert (a.blob - b.blob).abs().max() <= 2.1 * b.lr  # Adam moves an entry by about lr either way
        packed = b.packed.clone()
        b.pack()
        assert torch.equal(packed, b.packed)


def test_step_rejects_bad_arguments():
    tr = ranker.Trainer(np.ones(ia.RANKER_FLOATS, np.float32), batch=16)
    assert tr.lib.indialign_mlp_step(*[None] * 4, 16, 1.0, *[None] * 6, 1, 1e-3, 0.9, 0.999, 1e-8, *[None] * 3) < 0
