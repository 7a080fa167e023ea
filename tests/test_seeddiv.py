"""The FP64 quotients and square roots from FP32 seeds (csrc/seeddiv.cuh) and
the exact scalings and comparisons on the integer pipe, which the flux sweeps
use, must equal the IEEE-754 operations bit for bit: on the host against the
host's (C++ build of the same headers) and on the GPU against CUDA's."""
import os
import shutil
import subprocess

import pytest

import idefix_gb300 as ig

HERE = os.path.dirname(os.path.abspath(__file__))


def test_seeded_quotients_and_roots_match_host_ieee(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "seeddiv_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "native", "seeddiv_check.cpp")], check=True)
    r = subprocess.run([str(exe), "2000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip().startswith("0 mismatches")


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [5, 77])
def test_seeded_quotients_and_roots_match_cuda(seed):
    import ctypes

    from idefix_gb300 import build

    build.build_library()
    lib = ig.load_library()
    bad = ctypes.c_longlong(-1)
    assert lib.idfx_check_division(1 << 26, seed, ctypes.byref(bad)) == ig.OK
    assert bad.value == 0
