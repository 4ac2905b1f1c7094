"""The rounding bounds of the planar near / far split (rumdeed_gb300/csrc/rd_bounds.h)
hold for near lists of any length: sums of up to a million terms in the kernels' order,
with terms whose roundings agree.  And the guard of its decisions from FP32 targets holds
with every logarithm an ulp off either way, at a tip with parts that cancel too.  Compiled
for the host with g++."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_sums_stay_within_their_bounds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "near_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "near_check.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
