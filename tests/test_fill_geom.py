"""The NW fill's geometry as the kernels have it: csrc/fill_geom.h compiled for
the host, and the fill's schedule replayed with it (test_nw_fill replays it for
any choice of rows per lane)."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_nw_fill import Warp, direct, direction, fill

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "indialign_b200", "csrc")
PAD = 33

WRAP = """
#include "fill_geom.h"
extern "C" {
int pad() { return ia::kFillPad; }
void geom(int plen, int nlen, int W, int *o) {
    const ia::FillGeom g = ia::fill_geom(plen, nlen, W);
    o[0] = g.R; o[1] = g.S; o[2] = g.W; o[3] = g.G;
}
int trace_words(int np, int nn) { return (int)ia::fill_trace_words(np, nn); }
int column(int k, int half, int nlen) { return ia::fill_column(k, half, nlen); }
}
"""


@pytest.fixture(scope="module")
def geom_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("geom")
    src, so = d / "geom.cpp", d / "geom.so"
    src.write_text(WRAP)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("nlen", [0, 1, 2, 3, 64, 65])
def test_staged_columns_stay_inside_the_native_points(geom_lib, nlen):
    """Every pair that is staged, padding included; none is read of an empty side."""
    assert geom_lib.pad() == PAD
    pairs = (nlen + 1) >> 1
    for k in range(-PAD, pairs + PAD):
        for half in (0, 1):
            c = geom_lib.column(k, half, nlen)
            assert c < nlen, (k, half)
            if k < 0 or nlen == 0:
                assert c == -1
            else:
                assert c == min(2 * k + half, nlen - 1) >= 0


def _geom(lib, plen, nlen, W):
    o = (ctypes.c_int * 4)()
    lib.geom(plen, nlen, W, o)
    return dict(zip("RSWG", o))


# rows per lane (4 or 3, as the header chooses), stripes fewer than, as many as
# and more than the warps, last stripes of one row, odd and even column counts
SIZES = [(3, 3, 1, 3, 1, 0.0), (5, 40, 4, 3, 1, -0.6), (97, 21, 1, 4, 1, 0.0), (129, 20, 1, 3, 2, -0.6),
         (193, 21, 1, 4, 2, 0.0), (257, 36, 1, 3, 3, -0.6), (385, 33, 1, 4, 4, -0.6), (97, 131, 4, 4, 1, 0.0),
         (190, 36, 4, 3, 2, -0.6), (288, 51, 4, 3, 3, 0.0), (384, 20, 4, 4, 3, -0.6), (385, 130, 4, 4, 4, -0.6),
         (512, 35, 4, 4, 4, 0.0), (513, 21, 4, 3, 6, -0.6), (577, 36, 4, 3, 7, 0.0), (673, 21, 4, 3, 8, -1.0),
         (769, 21, 4, 4, 7, -0.6)]


@pytest.mark.parametrize("plen,nlen,W,R,S,gap", SIZES)
def test_fill_by_the_header_equals_a_row_by_row_fill(geom_lib, plen, nlen, W, R, S, gap):
    g = _geom(geom_lib, plen, nlen, W)
    assert (g["R"], g["S"], g["W"]) == (R, S, W)
    M = np.random.default_rng(plen * 1000 + nlen).integers(0, 5, (plen, nlen)) / 4.0
    mem, want = fill(M, gap, g), direct(M, gap)
    assert all(direction(mem, g, i, j) == d for (i, j), d in want.items())


def test_warps_by_the_header_never_wait_in_a_circle(geom_lib):
    """The shared fill's shapes by their step counts, and every trace inside the block that the host sizes."""
    for plen in (1, 32, 65, 96, 97, 129, 257, 289, 385, 513, 577, 673, 769, 1100, 2100):
        for nlen in (1, 2, 30, 31, 64, 99, 160, 161, 319, 321, 640, 1001):
            for W in (1, 4):
                g = _geom(geom_lib, plen, nlen, W)
                assert g["S"] * g["R"] * 64 * g["G"] <= geom_lib.trace_words(plen, nlen)
                assert g["S"] * g["R"] * 32 >= plen > (g["S"] - 1) * g["R"] * 32
                prog = [0] * W
                warps = [Warp(np.broadcast_to(0.0, (plen, nlen)), 0.0, g, w, {}, [], prog, 0) for w in range(W)]
                while any(x.todo for x in warps):
                    moved = False
                    for x in warps:
                        while x.todo and x.ready():
                            x.publish()
                            moved = True
                    assert moved, (plen, nlen, W)
