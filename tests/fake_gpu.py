"""The library's host code on a stand-in for the CUDA runtime
(native/fake_cudart.cpp): launches are written down instead of run and a chosen
allocation fails.  For tests of what the host code does; nothing is computed."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def build(tmp_path):
    """the library's objects linked with the stand-in"""
    from idefix_gb300 import build as b

    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    b.build_library()
    objs = [os.path.join(b.BUILD, os.path.splitext(s)[0] + ".o") for s in b.SOURCES]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(b.nvcc()))), "include")
    out = str(tmp_path / "libfake.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", include, "-o", out,
                    os.path.join(HERE, "native", "fake_cudart.cpp"), *objs, "-Wl,-Bsymbolic"], check=True)
    return out


class Fake:
    """idefix_gb300 with the stand-in library loaded in the place of the real one"""

    def __init__(self, tmp_path, monkeypatch):
        import idefix_gb300 as ig

        monkeypatch.setattr(ig, "_lib", None)
        self.ig = ig
        self.lib = ig.load_library(build(tmp_path))
        self.lib.fake_launches.restype = ctypes.c_char_p
        self.lib.fake_live_bytes.restype = ctypes.c_longlong

    def fail_in(self, n):
        """the n-th allocation from now on fails (0: the next one; -1: none)"""
        self.lib.fake_fail_in(n)

    def launches(self):
        """the launches since the last call, one a line"""
        return self.lib.fake_launches().decode().splitlines()

    def live_bytes(self):
        return self.lib.fake_live_bytes()
