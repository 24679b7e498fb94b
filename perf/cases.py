"""The work a user of this library has it do, as cases that can be timed: the
TM-score superposition search on host pairs and on CUDA tensors, plain and with
the learned seed ranker, from one short pair to large mixed-length batches; the
collection of ranker training data; and the ranker's training step and
prediction.

A case is a dict of plain values.  Its "kind":

  search   indialign_b200.search on host arrays
  tensors  indialign_b200.search_tensors on padded CUDA tensors
  collect  indialign_b200.collect_windows (plain search + labelled candidates)
  train    ranker.Trainer.step (forward, loss, backward, Adam, repack)
  predict  ranker.Trainer.predict

Structures are C1' traces of hairpin stems and loops (workloads.make_trace);
a pair's native is a noisy, rotated and translated copy of its prediction, or,
for "hard" pairs, another fold that keeps some of its stems.
"""
import math

import numpy as np
import torch

import indialign_b200 as ia
from indialign_b200 import ranker, workloads

F, H = ia.FEATURES, ranker.HIDDEN


def listed():
    return [
        # one short pair, all residues valid: what an interactive user scores; launches and latency
        {"name": "pair_64", "kind": "search", "n": 1, "lo": 64, "hi": 64, "sigma_lo": 2.0, "sigma_hi": 2.0,
         "invalid": 0.0, "hard": False, "learned": False},
        # one ribosomal-size pair of different folds: every rescue pass runs, nothing else fills the GPU
        {"name": "pair_hard_1203", "kind": "search", "n": 1, "lo": 1203, "hi": 1203, "sigma_lo": 6.0,
         "sigma_hi": 6.0, "invalid": 0.05, "hard": True, "learned": False},
        # a structure-prediction round's candidates for short targets, from host memory
        {"name": "short_64", "kind": "search", "n": 64, "lo": 40, "hi": 300, "sigma_lo": 0.5, "sigma_hi": 14.0,
         "invalid": 0.05, "hard": False, "learned": False},
        # an uneven batch of unlike folds (lengths log-uniform), from host memory
        {"name": "hard_48", "kind": "search", "n": 48, "lo": 30, "hi": 1500, "sigma_lo": 0.5, "sigma_hi": 14.0,
         "invalid": 0.05, "hard": True, "learned": False},
        # exhaustive scoring of a mixed-length batch that already is on the GPU
        {"name": "mixed_160", "kind": "tensors", "n": 160, "lo": 40, "hi": 1000, "sigma_lo": 0.5, "sigma_hi": 14.0,
         "invalid": 0.05, "hard": False, "learned": False, "dtype": "float64"},
        # the learned search of a small batch of FP32 coordinates, as a torch scorer holds them
        {"name": "learned_61", "kind": "tensors", "n": 61, "lo": 40, "hi": 700, "sigma_lo": 0.5, "sigma_hi": 14.0,
         "invalid": 0.05, "hard": False, "learned": True, "dtype": "float32"},
        # the learned search of a serving-size batch: the throughput configuration
        {"name": "learned_1024", "kind": "tensors", "n": 1024, "lo": 40, "hi": 1000, "sigma_lo": 0.5,
         "sigma_hi": 14.0, "invalid": 0.05, "hard": False, "learned": True, "dtype": "float64"},
        # the learned search of unlike folds, from host memory
        {"name": "learned_hard_64", "kind": "search", "n": 64, "lo": 30, "hi": 1500, "sigma_lo": 0.5,
         "sigma_hi": 14.0, "invalid": 0.05, "hard": True, "learned": True},
        # labelled candidates of a training chunk
        {"name": "collect_24", "kind": "collect", "n": 24, "lo": 40, "hi": 300, "sigma_lo": 0.5, "sigma_hi": 14.0,
         "invalid": 0.0, "hard": False},
        # one step of ranker training at its default batch
        {"name": "train_8192", "kind": "train", "rows": 8192},
        # the ragged last batch of an epoch
        {"name": "train_1003", "kind": "train", "rows": 1003},
        # predicted scores of a held-out set's candidates
        {"name": "predict_200k", "kind": "predict", "rows": 200003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "tensors", "tensors", "tensors", "collect", "train", "predict"])
    if kind == "train":
        return {"kind": "train", "rows": _log_int(rng, 63, 8192)}
    if kind == "predict":
        return {"kind": "predict", "rows": _log_int(rng, 999, 200003)}
    learned = kind != "collect" and rng.random() < 0.5
    hi = _log_int(rng, 60, 300 if kind == "collect" else 1000)
    # pairs so that the batch costs no more than the largest listed one of its kind
    most = 1024 if learned else 160
    room = (2.0e8 if learned else 3.0e7) if kind != "collect" else 7.0e5
    n = _log_int(rng, 1, max(2, min(most, int(room / (hi * hi)))))
    lo = rng.randint(30, hi)
    sigma = rng.uniform(0.5, 10.0)
    c = {"kind": kind, "n": n, "lo": lo, "hi": hi, "sigma_lo": round(sigma, 3),
         "sigma_hi": round(rng.uniform(sigma, 14.0), 3), "invalid": 0.0 if kind == "collect" else rng.choice([0.0, 0.05, 0.05]),
         "hard": kind == "search" and n <= 64 and rng.random() < 0.4}
    if kind != "collect":
        c["learned"] = learned
    if kind == "tensors":
        c["dtype"] = rng.choice(["float64", "float32"])
    return c


def _lengths(c):
    """The pairs' lengths belong to the case (a collection's outputs are sized by them)."""
    rng = np.random.default_rng([c["n"], c["lo"], c["hi"]])
    lo, hi = c["lo"], c["hi"]
    if c["hard"] and hi / lo > 10:
        return [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(c["n"])]
    return [int(rng.integers(lo, hi + 1)) for _ in range(c["n"])]


def _pairs(c, seed):
    """The case's pairs.  Predictions are windows of a few long traces (so that
    a large batch is made quickly); hard pairs are made one by one."""
    rng = np.random.default_rng(seed)
    n, lo, hi = c["n"], c["lo"], c["hi"]
    lens = _lengths(c)
    pool = None if c["hard"] else [workloads.make_trace(hi, rng) for _ in range(min(n, 16))]
    out = []
    for i, L in enumerate(lens):
        sigma = float(rng.uniform(c["sigma_lo"], c["sigma_hi"]))
        if c["hard"]:
            out.append(workloads.make_pair(L, sigma, rng, c["invalid"], hard=i % 2 == 0))
            continue
        a = int(rng.integers(0, hi - L + 1))
        pred = np.ascontiguousarray(pool[i % len(pool)][a:a + L])
        native = pred + rng.standard_normal((L, 3)) * sigma
        native = native @ workloads.random_rotation(rng).T + rng.uniform(-50, 50, 3)
        pv, nv = ((rng.uniform(size=L) >= c["invalid"]).astype(np.uint8) for _ in range(2))
        out.append(workloads.Pair(pred, np.ascontiguousarray(native), pv & nv, pv, nv, float(L), sigma))
    return out


def _training_rows(c, seed):
    """Standardised-looking candidate features, labels in 0..1 and a network
    as it is at the start of training."""
    rng = np.random.default_rng(seed)
    n = c["rows"]
    mean, std = rng.uniform(-1, 1, F).astype(np.float32), rng.uniform(0.2, 2, F).astype(np.float32)
    x = (rng.standard_normal((n, F)) * std + mean).astype(np.float32)
    return x, rng.uniform(0, 1, n).astype(np.float32), ranker.init_blob(mean, std, seed & 0x7FFFFFFF)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "predict"):
        x, t, blob = _training_rows(case, seed)
        tr = ranker.Trainer(blob, batch=case["rows"] if kind == "train" else 8192)
        return {"kind": kind, "trainer": tr, "x": torch.tensor(x, device="cuda"), "t": torch.tensor(t, device="cuda")}
    pairs = _pairs(case, seed)
    s = {"kind": kind, "ranker": ranker.default_weights() if case.get("learned") else None}
    if kind != "tensors":
        s["pairs"] = pairs
        return s
    N = max(p.pred.shape[0] for p in pairs)
    pred, nat = np.zeros((2, len(pairs), N, 3))
    v, pv, nv = np.zeros((3, len(pairs), N), np.uint8)
    for i, p in enumerate(pairs):
        L = p.pred.shape[0]
        pred[i, :L], nat[i, :L], v[i, :L], pv[i, :L], nv[i, :L] = p.pred, p.native, p.valid, p.pred_valid, p.native_valid
    dt = getattr(torch, case["dtype"])
    put = lambda a, d: torch.tensor(a, dtype=d, device="cuda")  # noqa: E731
    s.update(pred=put(pred, dt), native=put(nat, dt), valid=put(v, torch.uint8), pred_valid=put(pv, torch.uint8),
             native_valid=put(nv, torch.uint8), lengths=np.array([p.pred.shape[0] for p in pairs], np.int32))
    return s


def run(s):
    kind = s["kind"]
    if kind == "search":
        score, R, t = ia.search(s["pairs"], ranker=s["ranker"])
        return {"score": score, "R": R, "t": t}
    if kind == "tensors":
        score, R, t = ia.search_tensors(s["pred"], s["native"], s["valid"], s["pred_valid"], s["native_valid"],
                                        lengths=s["lengths"], ranker=s["ranker"])
        return {"score": score, "R": R, "t": t}
    if kind == "collect":
        (score, R, t), feat, label, off = ia.collect_windows(s["pairs"])
        feat[np.isnan(label)] = 0  # rows of candidates that were not refined carry no features
        return {"score": score, "R": R, "t": t, "feat": feat, "label": label, "off": off}
    if kind == "train":
        tr = s["trainer"]
        loss = tr.step(s["x"], s["t"])
        return {"loss": loss, "grad": tr.grad, "blob": tr.blob, "m": tr.m, "v": tr.v}
    return {"y": s["trainer"].predict(s["x"])}


def work(case):
    """Inputs read and outputs written once.  Operations of a search: the
    alignments that every pair gets whatever its score (two secondary-structure
    seeds, three dp_refine runs of two gap chains and the offset starts of two,
    18 per matrix cell) and the fragment seed bank (about 300 seeds of 11
    cutoffs, at least three sweeps of 55 per residue); weak pairs need more."""
    if case["kind"] in ("train", "predict"):
        n, p = case["rows"], ia.RANKER_FLOATS
        once = 2.0 * n * (F * H + H * H + H)
        if case["kind"] == "predict":
            return {"bytes": n * (F + 1) * 4 + p * 4, "flops": once}
        return {"bytes": n * (F + 1) * 4 + p * 4 * 7, "flops": 3 * once}
    lens = _lengths(case)
    return {"bytes": sum(51 * L + 104 for L in lens), "flops": sum(28.0 * 18 * L * L + 300 * 11 * 3 * 55 * L for L in lens)}


def exact(case, seed):
    """The ranker's training step and prediction in 64 bits.  A search has no
    such value at hand: its result is what the heuristic's many thousand
    alignments and refinements arrive at, hours of plain array code."""
    if case["kind"] not in ("train", "predict"):
        return None
    x, t, blob = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in _training_rows(case, seed))
    blob.requires_grad_(True)
    r = ranker
    part = lambda a, b, *s: blob[a:b].reshape(*s)  # noqa: E731
    mean, std = blob[r.MEAN:r.STD].detach(), blob[r.STD:r.W1].detach()
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
    h = gelu((x - mean) / std @ part(r.W1, r.B1, F, H) + part(r.B1, r.W2, H))
    h = gelu(h @ part(r.W2, r.B2, H, H) + part(r.B2, r.W3, H))
    y = h @ part(r.W3, r.B3, H) + blob[r.B3]
    if case["kind"] == "predict":
        return {"y": y.detach()}
    m = y.shape[0] // 2
    ya, yb, ta, tb = y[:2 * m:2], y[1:2 * m:2], t[:2 * m:2], t[1:2 * m:2]
    sign = torch.sign(ta - tb) * ((ta - tb).abs() > 1e-6)
    rank = torch.nn.functional.softplus(-sign * (ya - yb)) * sign.abs()
    loss = ((y - t) ** 2).mean() + rank.sum() / max(m, 1)  # Trainer's default weight of the ranking term: 1
    (g,) = torch.autograd.grad(loss, blob)
    # Adam's first step with the trainer's defaults; mean and std are not trained
    mom, var = 0.1 * g, 0.001 * g * g
    step = 1e-3 * g / (g.abs() + 1e-8)
    return {"loss": loss.detach().reshape(1), "grad": g, "blob": (blob - step).detach(), "m": mom, "v": var}
