"""The NW fill's geometry as the kernels have it: csrc/fill_geom.h compiled for
the host."""
from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "indialign_b200", "csrc")
PAD = 33

WRAP = """
#include "fill_geom.h"
extern "C" {
int pad() { return ia::kFillPad; }
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
