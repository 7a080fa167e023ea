"""HLLD's degeneracy tests (csrc/exact_ops.cuh), decided in FP32 where the
margin is clear, must agree with the FP64 comparisons at every magnitude of the
wave speeds, FP32's subnormal range and below it included."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_degeneracy_tests_match_fp64_at_every_magnitude(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "degenerate_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "degenerate_check.cpp")], check=True)
    r = subprocess.run([str(exe), "3000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
