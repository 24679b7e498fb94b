"""CPU replay of the NW fill's schedule (csrc/nw_fill.cuh, fill_geom.h): the
wavefront of R rows x 2 columns per lane and step, the trace words, the
boundary rows between stripes, and W warps sharing one alignment.

Checked: every access lies inside the trace block, the staged columns and the
boundary rows that the host sizes; boundary pairs are read after they were
written; the warps never wait for one another in a circle; and the directions
read back from the words are those of a row-by-row fill of the same matrix."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

LAG, PAD = 49, 33


def geom(plen, nlen, W, R=None):
    """fill_geom; with R given, that choice of rows per lane."""
    n32, np_ = (plen + 31) >> 5, (nlen + 1) >> 1
    best = None
    for r in (4, 3, 2) if R is None else (R,):
        S = (n32 + r - 1) // r
        cost = ((S + W - 1) // W * (np_ + 31) + (min(S, W) - 1) * LAG) * (20 + 32 * r)
        if best is None or cost < best[0]:
            best = (cost, r, S)
    return {"R": best[1], "S": best[2], "W": W, "G": (np_ + 46) // 16}


def trace_words(np_, nn):
    return ((np_ + 31) // 32 + 3) * 64 * (((nn + 1) // 2 + 46) // 16)


def cell(ds, sc, up, left, gap):
    """fill_cell; a NaN score (left of the matrix) leaves max(left, up)."""
    diag = ds + sc
    m = max(left, up)
    isd = diag >= m
    h = diag if isd else m
    return h, diag + gap if isd else m, int(not isd), int(left < up)


class Warp:
    """nw_fill of one warp, as a generator of its 16-step groups."""

    def __init__(self, M, gap, g, w, mem, bnd, prog, size):
        self.M, self.gap, self.g, self.w, self.mem, self.bnd, self.prog, self.size = M, gap, g, w, mem, bnd, prog, size
        self.np = (M.shape[1] + 1) >> 1
        self.todo = [(k, t0) for k in range(w, g["S"], g["W"]) for t0 in range(0, self.steps(k), 16)]

    def steps(self, k):
        last = (self.M.shape[0] - 1 - k * 32 * self.g["R"]) // self.g["R"] if k == self.g["S"] - 1 else 31
        return self.np + last

    def ready(self):
        k, t0 = self.todo[0]
        W, w = self.g["W"], self.w
        if W == 1 or k == 0:
            return True
        need = (k // W if w > 0 else k // W - 1) * (self.np + 64) + min(t0 + 17, self.np)
        return self.prog[w - 1 if w > 0 else W - 1] >= need

    def publish(self):
        k, t0 = self.todo.pop(0)
        self.prog[self.w] = k // self.g["W"] * (self.np + 64) + max(min(t0 + 16, self.steps(k)) - 31, 0)

    def boundary(self, k, s):
        assert -PAD <= s < self.np + PAD
        if s >= self.np:
            return (7.0,) * 4  # never reaches the matrix
        v, src = self.bnd[(k - 1) % self.g["W"]][s]
        assert src == k - 1, "boundary of another stripe"
        return v

    def group(self):
        g, M, gap, w = self.g, self.M, self.gap, self.w
        plen, nlen = M.shape
        R, S = g["R"], g["S"]
        k, t0 = self.todo[0]
        if t0 == 0:
            z = lambda: [0.0] * R  # noqa: E731
            self.L = [dict(h=z(), hp=z(), ta=[0] * R, tb=[0] * R, upprev=0.0, hb=(0.0, 0.0), pb=(0.0, 0.0))
                      for _ in range(32)]
            self.bn = self.boundary(k, 0) if k > 0 else (0.0,) * 4
        n16 = min(16, self.steps(k) - t0)
        for u in range(n16):
            old = [(c["hb"], c["pb"]) for c in self.L]
            out = None
            for l, c in enumerate(self.L):
                (up0, up1), (pu0, pu1) = old[max(l - 1, 0)]
                if l == 0:
                    up0, pu0, up1, pu1 = self.bn
                s = t0 + u - l
                assert -PAD <= s < self.np + PAD
                row0 = (k * 32 + l) * R
                c0, c1 = min(2 * s, nlen - 1), min(2 * s + 1, nlen - 1)
                e = [(M[min(row0 + r, plen - 1), c0], M[min(row0 + r, plen - 1), c1]) if s >= 0 else (np.nan, np.nan)
                     for r in range(R)]
                n0, p0, nh, nhp = [0.0] * R, [0.0] * R, [0.0] * R, [0.0] * R
                for col, (h, hp) in enumerate(((n0, p0), (nh, nhp))):
                    for r in range(R):
                        ds = (c["upprev"], up0)[col] if r == 0 else (c["h"], n0)[col][r - 1]
                        h[r], hp[r], a, b = cell(ds, e[r][col], (pu0, pu1)[col] if r == 0 else hp[r - 1],
                                                 (c["hp"], p0)[col][r], gap)
                        c["ta"][r], c["tb"][r] = (c["ta"][r] << 1 | a) & 0xFFFFFFFF, (c["tb"][r] << 1 | b) & 0xFFFFFFFF
                c["h"], c["hp"], c["upprev"] = nh, nhp, up1
                c["hb"], c["pb"] = (n0[R - 1], nh[R - 1]), (p0[R - 1], nhp[R - 1])
                if l == 31 and k + 1 < S:
                    assert s < self.np + PAD
                    out = (s, (n0[R - 1], p0[R - 1], nh[R - 1], nhp[R - 1]))
            if k > 0:
                self.bn = self.boundary(k, t0 + u + 1)
            if out:
                self.bnd[w][out[0]] = (out[1], k)
        for l, c in enumerate(self.L):
            if (k * 32 + l) * R < plen:
                at = ((k * g["G"] + t0 // 16) * 32 + l) * 2 * R
                for r in range(R):
                    for p, word in ((0, c["ta"][r]), (1, c["tb"][r])):
                        assert 0 <= at + 2 * r + p < self.size
                        self.mem[at + 2 * r + p] = (word << 2 * (16 - n16)) & 0xFFFFFFFF
            c["ta"], c["tb"] = [0] * R, [0] * R
        self.publish()


def fill(M, gap, g):
    """The trace words of the fill: warps advance in turn, as far as their waits let them."""
    size = trace_words(*M.shape)
    mem, bnd, prog = {}, [{} for _ in range(g["W"])], [0] * g["W"]
    warps = [Warp(M, gap, g, w, mem, bnd, prog, size) for w in range(g["W"])]
    while any(x.todo for x in warps):
        moved = False
        for x in reversed(warps):
            if x.todo and x.ready():
                x.group()
                moved = True
        assert moved, "the warps wait for one another"
    return mem


def direction(mem, g, i, j):
    R = g["R"]
    k, ri = (i - 1) // (32 * R), (i - 1) % (32 * R)
    l, rr = ri // R, ri % R
    word = (l + ((j - 1) >> 1)) >> 4
    a = ((k * g["G"] + word) * 32 + l) * 2 * R + 2 * rr
    pos = 32 * word + 32 - 2 * l - j
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


SIZES = [(3, 3, 1, None, 0.0), (3, 3, 4, None, -0.6), (7, 41, 1, None, -0.6), (33, 31, 1, 2, 0.0), (64, 64, 1, 2, -0.6),
         (97, 20, 1, 3, 0.0), (129, 64, 1, 4, -0.6), (130, 101, 1, 2, -0.6), (100, 130, 1, 3, 0.0),
         (65, 66, 4, 2, -0.6), (330, 40, 4, 2, 0.0), (200, 90, 4, 2, -0.6), (520, 50, 4, 3, 0.0), (300, 35, 4, 2, -1.0)]


@pytest.mark.parametrize("plen,nlen,W,R,gap", SIZES)
def test_fill_equals_a_row_by_row_fill(plen, nlen, W, R, gap):
    M = np.random.default_rng(plen * 1000 + nlen).integers(0, 5, (plen, nlen)) / 4.0
    g = geom(plen, nlen, W, R)
    mem, want = fill(M, gap, g), direct(M, gap)
    assert all(direction(mem, g, i, j) == d for (i, j), d in want.items())


def test_warps_never_wait_in_a_circle():
    """Every shape of the shared fill, by its step counts alone."""
    for plen in (1, 65, 129, 300, 513, 700, 1100, 2100):
        for nlen in (1, 2, 30, 31, 64, 99, 160, 161, 319, 321, 640, 1001):
            for R in (2, 3, 4):
                g = geom(plen, nlen, 4, R)
                prog = [0] * 4
                warps = [Warp(np.broadcast_to(0.0, (plen, nlen)), 0.0, g, w, {}, [], prog, 0) for w in range(4)]
                while any(x.todo for x in warps):
                    moved = False
                    for x in warps:
                        while x.todo and x.ready():
                            x.publish()
                            moved = True
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
