"""The bench line's DRAM traffic is scaled from captures of the present build,
not from the earlier ones that roofline_record falls back on."""
from __future__ import annotations

import ast
import inspect
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


def test_main_uses_the_present_captures():
    """18.872 GB over 21.9986 G NW cells; 639.0 MB over 11.221 G residue visits."""
    calls = [n for n in ast.walk(ast.parse(inspect.getsource(bench.main))) if isinstance(n, ast.Call)
             and getattr(n.func, "id", "") == "roofline_record"]
    assert calls and all(ast.unparse(c.args[-1]) == "DRAM_BYTES" for c in calls)
    assert bench.DRAM_BYTES["k_chain"] == pytest.approx(0.8579, rel=1e-3)
    assert bench.DRAM_BYTES["k_bank"] == pytest.approx(0.05695, rel=1e-3)
