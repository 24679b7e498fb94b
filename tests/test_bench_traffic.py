"""The bench line's DRAM traffic is scaled from captures of the present build
(profiles/kernels_b200.md), not from the earlier ones that roofline_record falls
back on."""
from __future__ import annotations

import ast
import inspect
import os
import re
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_traffic_follows_the_given_capture():
    kern = [600.0, 750.0, 0.0, 0.0, 120.0]
    ctr = [2.0e10, 1.0e9, 2.5e11, 0, 0, 0, 0, 150, 3.0, 1.0, 0.0, 0.0]
    k = bench.roofline_record(kern, ctr, 1400.0, 67.5, "measured", bench.DRAM_BYTES)["kernels"]
    assert k["k_chain"]["traffic"] == pytest.approx(bench.DRAM_BYTES["k_chain"] * 2.0e10)
    assert k["k_bank"]["traffic"] == pytest.approx(bench.DRAM_BYTES["k_bank"] * 2.5e11)


def test_main_uses_the_captures_that_the_profile_states():
    calls = [n for n in ast.walk(ast.parse(inspect.getsource(bench.main))) if isinstance(n, ast.Call)
             and getattr(n.func, "id", "") == "roofline_record"]
    assert calls and all(ast.unparse(c.args[-1]) == "DRAM_BYTES" for c in calls)
    text = open(os.path.join(ROOT, "profiles", "kernels_b200.md")).read()
    for name, unit in (("k_chain", "NW cell"), ("k_bank", "residue visit")):
        m = re.search(rf"`{name}`: ([0-9.]+) bytes per {unit}", text)
        assert m and float(m.group(1)) == pytest.approx(bench.DRAM_BYTES[name], rel=1e-3)
