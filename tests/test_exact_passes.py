"""Halved sums, quarters, upwind terms, products by powers of two and HLLD's
degeneracy tests of the FP64 kernels (csrc/exact_ops.cuh) must equal the IEEE-754 expressions bit for bit over
random bit patterns, zeros, subnormals, infinities and NaNs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_pass_helpers_match_host_ieee(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "passes_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "passes_check.cpp")], check=True)
    r = subprocess.run([str(exe), "2000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip().startswith("0 mismatches")
