"""CPU replay of the NW fill's schedule (csrc/nw_fill.cuh, fill_geom.h): the
wavefront of R rows x 2 columns per lane and step, the trace words, the
boundary rows between stripes, and W warps sharing one alignment.

Checked: every store lies inside the trace block that the host sizes
(fill_trace_words); every boundary pair is read after it was written, across a
16-step group boundary; the warps never wait for one another in a circle; and
the directions and the path read back from the words are those of a row-by-row
fill of the same matrix."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

LAG = 49


def min_period(W):
    return 32 * W + 32 if W > 1 else 50


def geom(plen, nlen, W, R=None):
    """fill_geom; with R given, that choice of rows per lane."""
    n32, np_ = (plen + 31) >> 5, (nlen + 1) >> 1
    best = None
    for r in (4, 3, 2, 1) if R is None else (R,):
        S = (n32 + r - 1) // r
        rounds = (S + W - 1) // W
        P2 = min_period(W) if rounds > 1 and np_ < min_period(W) else np_
        cost = (rounds * P2 + (min(S, W) - 1) * LAG + 31) * (25 + 34 * r)
        if best is None or cost < best[0]:
            best = (cost, r, S, P2)
    _, r, S, P2 = best
    return {"R": r, "S": S, "W": W, "P2": P2, "G": (P2 + 45) // 16 + 1}


def trace_words(np_, nn):
    P2 = max((nn + 1) // 2, min_period(4))
    return ((np_ + 31) // 32 + 3) * 64 * ((P2 + 45) // 16 + 1)


def cell(ds, sc, up, left, gap):
    diag = ds + sc
    m = max(left, up)
    h = max(diag, m)
    hp = (diag + gap if diag >= m else m) if gap else h
    return h, hp, int(diag < m), int(left < up)


class Warp:
    """The state of nw_fill for one warp, advanced one 16-step group at a time."""

    def __init__(self, M, gap, g, w, mem, bnd, prog, size):
        self.M, self.gap, self.g, self.w, self.mem, self.bnd, self.prog, self.size = M, gap, g, w, mem, bnd, prog, size
        plen, nlen = M.shape
        R, S, W, P2 = g["R"], g["S"], g["W"], g["P2"]
        self.np = (nlen + 1) >> 1
        self.nq = (S - w + W - 1) // W if S > w else 0
        k_last = w + (self.nq - 1) * W
        last = (plen - 1 - k_last * 32 * R) // R if k_last == S - 1 else 31
        self.total = (self.nq - 1) * P2 + last + self.np if self.nq else 0
        self.t0, self.tq, self.qn, self.slot = 0, 0, 0, None
        z = lambda: [0.0] * R  # noqa: E731
        self.L = [dict(s=P2 - l, q=-1, ok=False, wlim=0, rlim=0, wp=0, h=z(), hp=z(), ta=[0] * R, tb=[0] * R, upprev=0.0,
                       hb=(0.0, 0.0), pb=(0.0, 0.0), bn=None, row0=None) for l in range(32)]

    def done(self):
        return self.t0 >= self.total

    def ready(self):
        """The wait at a group's start (W > 1)."""
        g = self.g
        if g["W"] == 1:
            return True
        P2 = g["P2"]
        ql, sl = self.t0 // P2, self.t0 % P2 + 16
        if sl >= P2:
            ql, sl = ql + 1, sl - P2
        if ql >= self.nq:
            ql, sl = self.nq - 1, self.np
        qp, wprod = (ql, self.w - 1) if self.w > 0 else (ql - 1, g["W"] - 1)
        return qp < 0 or self.prog[wprod] >= qp * P2 + 32 + min(sl, self.np - 1)

    def store(self, c, sh):
        R = self.g["R"]
        for r in range(R):
            for p, word in ((0, c["ta"][r]), (1, c["tb"][r])):
                a = c["wp"] + 2 * r + p
                assert 0 <= a < self.size
                self.mem[a] = (word << sh) & 0xFFFFFFFF

    def read_boundary(self, k, s, stamp):
        (h0, p0, h1, p1), src, wrote = self.bnd[(k - 1) % self.g["W"]][s]
        assert src == k - 1, "boundary of another stripe"
        # same warp: written in an earlier group; another warp: before its published count
        assert wrote < self.t0 if self.g["W"] == 1 else wrote < self.prog[(k - 1) % self.g["W"]]
        return h0, p0, h1, p1

    def group(self):
        g, M, gap = self.g, self.M, self.gap
        plen, nlen = M.shape
        R, S, W, P2, w = g["R"], g["S"], g["W"], g["P2"], self.w
        t0 = self.t0
        if self.tq < t0 + 16 and self.qn < self.nq:
            for c in self.L:  # nobody still has to load the slot's old content
                assert self.slot is None or c["q"] >= self.slot
            self.slot = self.qn
            self.tq += P2
            self.qn += 1
        n16 = min(16, self.total - t0)
        for u in range(n16):
            old = [(c["hb"], c["pb"]) for c in self.L]
            writes = []
            for l, c in enumerate(self.L):
                (up0, up1), (pu0, pu1) = old[max(l - 1, 0)]
                if c["s"] == P2:
                    if c["ok"] and u > 0:
                        self.store(c, 2 * (16 - u))
                    c["s"], c["q"] = 0, c["q"] + 1
                    k = w + c["q"] * W
                    c["row0"] = (k * 32 + l) * R
                    c["ok"] = c["q"] < self.nq and c["row0"] < plen
                    if c["ok"]:
                        assert self.slot == c["q"]
                    c["h"], c["hp"], c["ta"], c["tb"], c["upprev"] = [0.0] * R, [0.0] * R, [0] * R, [0] * R, 0.0
                    c["wp"] = ((k * g["G"] + ((t0 + u) >> 4) - ((c["q"] * P2) >> 4)) * 32 + l) * 2 * R
                    c["wlim"] = self.np if l == 31 and c["ok"] and k + 1 < S else 0
                    c["rlim"] = self.np if l == 0 and c["ok"] and k > 0 else 0
                    c["bn"] = self.read_boundary(k, 0, t0 + u) if c["rlim"] else (0.0,) * 4
                if l == 0:
                    up0, pu0, up1, pu1 = c["bn"]
                s = c["s"]
                if 0 <= s + 1 < c["rlim"]:
                    c["bn"] = self.read_boundary(w + c["q"] * W, s + 1, t0 + u)
                sc = s if 0 <= s < self.np else self.np - 1
                rows = [min((c["row0"] or 0) + r, plen - 1) for r in range(R)]
                c0, c1 = 2 * sc, min(2 * sc + 1, nlen - 1)
                n0, p0 = [0.0] * R, [0.0] * R
                hold = list(c["h"])
                for r in range(R):
                    n0[r], p0[r], a, b = cell(c["upprev"] if r == 0 else hold[r - 1], M[rows[r], c0],
                                              pu0 if r == 0 else p0[r - 1], c["hp"][r], gap)
                    c["ta"][r], c["tb"][r] = (c["ta"][r] << 1 | a) & 0xFFFFFFFF, (c["tb"][r] << 1 | b) & 0xFFFFFFFF
                nh, nhp = [0.0] * R, [0.0] * R
                for r in range(R):
                    nh[r], nhp[r], a, b = cell(up0 if r == 0 else n0[r - 1], M[rows[r], c1],
                                               pu1 if r == 0 else nhp[r - 1], p0[r], gap)
                    c["ta"][r], c["tb"][r] = (c["ta"][r] << 1 | a) & 0xFFFFFFFF, (c["tb"][r] << 1 | b) & 0xFFFFFFFF
                c["h"], c["hp"], c["upprev"] = nh, nhp, up1
                c["hb"], c["pb"] = (n0[R - 1], nh[R - 1]), (p0[R - 1], nhp[R - 1])
                if 0 <= s < c["wlim"]:
                    writes.append((s, (n0[R - 1], p0[R - 1], nh[R - 1], nhp[R - 1]), w + c["q"] * W))
                c["s"] += 1
            for s, v, k in writes:
                self.bnd[w][s] = (v, k, t0 + u)
        for c in self.L:
            if c["ok"]:
                self.store(c, 2 * (16 - n16))
            c["wp"] += 64 * R
            c["ta"], c["tb"] = [0] * R, [0] * R
        self.t0 += n16
        self.prog[w] = self.t0


def fill(M, gap, g):
    """The trace words of the fill: warps advance in turn, as far as their waits let them."""
    size = trace_words(*M.shape)
    mem, bnd, prog = {}, [{} for _ in range(g["W"])], [0] * g["W"]
    warps = [Warp(M, gap, g, w, mem, bnd, prog, size) for w in range(g["W"])]
    while not all(x.done() for x in warps):
        moved = False
        for x in reversed(warps):
            if not x.done() and x.ready():
                x.group()
                moved = True
        assert moved, "the warps wait for one another"
    return mem


def direction(mem, g, i, j):
    R, W = g["R"], g["W"]
    k, ri = (i - 1) // (32 * R), (i - 1) % (32 * R)
    l, rr, base = ri // R, ri % R, (k // W) * g["P2"]
    word = (base + l + ((j - 1) >> 1)) >> 4
    a = ((k * g["G"] + word - (base >> 4)) * 32 + l) * 2 * R + 2 * rr
    pos = 32 * word + 32 - 2 * (base + l) - j
    if not (mem[a] >> pos) & 1:
        return 0
    return 1 if (mem[a + 1] >> pos) & 1 else 2  # up : left


def direct(M, gap):
    plen, nlen = M.shape
    H, Hp = np.zeros((plen + 1, nlen + 1)), np.zeros((plen + 1, nlen + 1))
    out = {}
    for i in range(1, plen + 1):
        for j in range(1, nlen + 1):
            H[i, j], Hp[i, j], a, b = cell(H[i - 1, j - 1], M[i - 1, j - 1], Hp[i - 1, j], Hp[i, j - 1], gap)
            out[i, j] = 0 if not a else (1 if b else 2)
    return out


SIZES = [(3, 3, 1, None, 0.0), (3, 3, 4, None, -0.6), (7, 41, 1, None, -0.6), (33, 31, 1, 1, 0.0), (64, 64, 1, 2, -0.6),
         (97, 20, 1, 3, 0.0), (129, 64, 1, 4, -0.6), (130, 101, 1, 2, -0.6), (100, 130, 1, 1, 0.0),
         (65, 66, 4, 1, -0.6), (150, 40, 4, 1, 0.0), (200, 90, 4, 1, -0.6), (260, 50, 4, 2, 0.0), (300, 35, 4, 1, -1.0)]


@pytest.mark.parametrize("plen,nlen,W,R,gap", SIZES)
def test_fill_equals_a_row_by_row_fill(plen, nlen, W, R, gap):
    M = np.random.default_rng(plen * 1000 + nlen).integers(0, 5, (plen, nlen)) / 4.0
    g = geom(plen, nlen, W, R)
    mem, want = fill(M, gap, g), direct(M, gap)
    assert all(direction(mem, g, i, j) == d for (i, j), d in want.items())


def test_warps_never_wait_in_a_circle():
    """Every shape of the shared fill, by its step counts alone."""
    for plen in (1, 65, 129, 300, 513, 700, 1100, 2100):
        for nlen in (1, 2, 30, 31, 64, 99, 160, 161, 319, 320, 321, 640, 1001):
            for R in (1, 2, 3, 4):
                g = geom(plen, nlen, 4, R)
                M = np.broadcast_to(0.0, (plen, nlen))
                prog = [0] * 4
                warps = [Warp(M, 0.0, g, w, {}, [], prog, 0) for w in range(4)]
                while not all(x.done() for x in warps):
                    moved = False
                    for x in warps:
                        while not x.done() and x.ready():
                            x.t0 += min(16, x.total - x.t0)
                            prog[x.w], moved = x.t0, True
                    assert moved, (plen, nlen, R)
                assert g["S"] * g["R"] * 64 * g["G"] <= trace_words(plen, nlen)


def _path(M, gap):
    """Aligned pairs of the FP32 matrix M by the reference's rules, row by row in FP32."""
    plen, nlen = M.shape
    f = np.float32
    H, Hp = np.zeros((plen + 1, nlen + 1), f), np.zeros((plen + 1, nlen + 1), f)
    D = np.zeros((plen + 1, nlen + 1), np.int8)
    for s in range(2, plen + nlen + 1):  # anti-diagonals
        i = np.arange(max(1, s - nlen), min(plen, s - 1) + 1)
        j = s - i
        diag = H[i - 1, j - 1] + M[i - 1, j - 1]
        left, up = Hp[i, j - 1], Hp[i - 1, j]
        isd, lu = (diag >= up) & (diag >= left), left >= up
        H[i, j] = np.where(isd, diag, np.where(lu, left, up))
        Hp[i, j] = np.where(isd, diag + f(gap), H[i, j])
        D[i, j] = np.where(isd, 0, np.where(lu, 2, 1))
    out, i, j = [], plen, nlen
    while i > 0 and j > 0:
        if D[i, j] == 0:
            out.append((i - 1, j - 1))
        i, j = i - (D[i, j] != 2), j - (D[i, j] != 1)
    return out[::-1]


@pytest.mark.gpu
@pytest.mark.parametrize("warps", [1, 4])
@pytest.mark.parametrize("plen,nlen", [(3, 3), (5, 40), (31, 33), (64, 64), (65, 129), (130, 97), (200, 99),
                                       (385, 70), (300, 401), (640, 333)])
def test_gpu_fill_and_traceback(plen, nlen, warps):
    """Every score mode against the row-by-row path.  Coordinates on a coarse
    grid and power-of-two scales keep the distance arithmetic exact, so the
    matrices are equal bit for bit (and full of ties)."""
    import indialign_b200 as ia
    rng = np.random.default_rng(plen * 7 + nlen)
    P, Q = rng.integers(-12, 13, (plen, 3)) / 2.0, rng.integers(-12, 13, (nlen, 3)) / 2.0
    rt = np.array([0, 1, 0, -1, 0, 0, 0, 0, 1, 1.5, -2, 0.5], np.float64)
    lp, ln = rng.choice(list(b"L<>"), plen).astype(np.uint8), rng.choice(list(b"L<>"), nlen).astype(np.uint8)
    moved = P @ rt[:9].reshape(3, 3) + rt[9:]
    d2 = ((moved[:, None] - Q[None]) ** 2).sum(2).astype(np.float32)
    r = np.float32(1) / (np.float32(1) + d2 * np.float32(0.125))
    same = lp[:, None] == ln[None]
    dp = np.where(d2 <= np.float32(90), r, np.float32(0))
    f = ia.load().indialign_selftest_nw
    f.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] * 5 + [ctypes.c_int] + [ctypes.c_float] * 3 + [ctypes.c_int] + [ctypes.c_void_p] * 3
    for smode, gap, M in ((0, 0.0, dp), (0, np.float32(-0.6), dp), (1, -1.0, same.astype(np.float32)),
                          (2, -1.0, np.where(same, r + np.float32(0.5), r))):
        ap, an, na = np.zeros(min(plen, nlen), np.int32), np.zeros(min(plen, nlen), np.int32), np.zeros(1, np.int32)
        rc = f(plen, nlen, P.ctypes.data, Q.ctypes.data, rt.ctypes.data, lp.ctypes.data, ln.ctypes.data, smode, gap,
               0.125, 90.0, warps, ap.ctypes.data, an.ctypes.data, na.ctypes.data)
        assert rc == 0
        assert list(zip(ap[:na[0]], an[:na[0]])) == _path(M, gap), (smode, gap)


@pytest.mark.gpu
def test_gpu_reciprocal_is_correctly_rounded():
    import indialign_b200 as ia
    bad = ctypes.c_ulonglong(1)
    assert ia.load().indialign_selftest_rcp_f32(ctypes.byref(bad)) == 0
    assert bad.value == 0
