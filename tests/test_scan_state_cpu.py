"""The unit form's per-range scan state: whatever the order of the warp that publishes it and the
warp that reads it, a range is in the full form or has one of the two thresholds.  (Read as neither,
its next tiles would be searched by nobody and a better candidate there lost.)"""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FULL, NOTHING = -1.0, float("inf")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("scan_state") / "scan_state.so")
    res = subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-o", out,
                          os.path.join(ROOT, "tests", "scan_state_harness.cpp")],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    lib = C.CDLL(out)
    lib.scan_orders.argtypes = [C.c_float, C.c_float]
    return lib


@pytest.mark.parametrize("a,b", [(FULL, 64.0), (FULL, 4096.0), (64.0, 100.5), (100.5, FULL),
                                 (FULL, FULL), (NOTHING, FULL), (NOTHING, 64.0)])
def test_every_order_shows_one_of_the_states(harness, a, b):
    assert harness.scan_orders(a, b) >= 2
