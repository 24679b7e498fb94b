"""Trainer.step goes through its parts where they are overridden (gradient
clipping, a sum over ranks, another loss), and in one library call otherwise.
The library is a fake that notes the calls."""
from __future__ import annotations

import types

import pytest
import torch

from indialign_b200 import ranker


class FakeLib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name.removeprefix("indialign_mlp_"))
            return 0
        return call


def _trainer(cls):
    tr = cls.__new__(cls)
    tr.torch, tr.lib, tr.batch, tr.steps = torch, FakeLib(), 8, 0
    tr.lr, tr.lam, tr.beta1, tr.beta2, tr.eps = 1e-3, 1.0, 0.9, 0.999, 1e-8
    for k in ("blob", "m", "v", "grad", "packed", "save", "work", "y", "dy", "loss"):
        setattr(tr, k, torch.zeros(8))
    return tr


class Plain(ranker.Trainer):
    stream = None


class Clipped(Plain):
    def gradients(self, x, t):
        loss, grad = super().gradients(x, t)
        self.lib.calls.append("clip")
        return loss, grad


class OwnForward(Plain):
    def forward(self, x, save=False):
        self.lib.calls.append("own")
        return super().forward(x, save)


class OwnPack(Plain):
    def pack(self):
        super().pack()
        self.lib.calls.append("own")


PARTS = ["forward", "loss", "backward", "adam", "pack"]


@pytest.mark.parametrize("cls,want", [(Plain, ["step"]),
                                      (Clipped, PARTS[:3] + ["clip"] + PARTS[3:]),
                                      (OwnForward, ["own"] + PARTS),
                                      (OwnPack, PARTS + ["own"])])
def test_step_takes_the_parts_that_a_class_overrides(cls, want):
    tr = _trainer(cls)
    x, t = torch.zeros(4, 16), torch.zeros(4)
    assert tr.step(x, t) is tr.loss
    assert tr.lib.calls == want and tr.steps == 1


def test_step_takes_a_part_put_in_place(monkeypatch):
    x, t = torch.zeros(4, 16), torch.zeros(4)
    tr = _trainer(Plain)
    own = tr.gradients
    tr.gradients = types.MethodType(lambda self, x, t: (self.lib.calls.append("own"), own(x, t))[1], tr)
    tr.step(x, t)
    assert tr.lib.calls == ["own"] + PARTS
    tr = _trainer(Plain)
    whole = ranker.Trainer.gradients
    monkeypatch.setattr(ranker.Trainer, "gradients", lambda self, x, t: (self.lib.calls.append("own"), whole(self, x, t))[1])
    tr.step(x, t)
    assert tr.lib.calls == ["own"] + PARTS
