"""Learned boxes where the device has no room for the corrections of all three
directions or for the FP32 primitives: the block is made and run all the same,
window by window in the memory of the solver's own fields (the host code on a
stand-in for the CUDA runtime, and the windows' arithmetic on the host)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from fake_gpu import Fake

HERE = os.path.dirname(os.path.abspath(__file__))
N = (40, 36, 44)
NC = 44 * 40 * 48
NPARAM = 216 * 128 + 128 + 128 * 128 + 128 + 128 * 16 + 16


def test_windows_hold_every_cell_once(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "window_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-o", str(exe),
                    os.path.join(HERE, "native", "learned_window_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.fixture
def fake(tmp_path, monkeypatch):
    return Fake(tmp_path, monkeypatch)


def _run(fake, fail_create, fail_set):
    """(live bytes, names and grids of the learned launches of a cycle)"""
    ig = fake.ig
    fake.fail_in(fail_create)
    blk = ig.GpuBlock(3, N, order="learned", cfl=0.3, first_dt=1e-4)
    fake.fail_in(fail_set)
    blk.set_learned(np.zeros(NPARAM, np.float32))
    fake.fail_in(-1)
    live = fake.live_bytes()
    fake.launches()
    blk.run(max_cycles=1)
    out = [line for line in fake.launches() if "learned" in line]
    blk.close()
    assert fake.live_bytes() == 0
    return live, out


def test_learned_box_without_room(fake):
    whole, launches = _run(fake, -1, -1)
    assert len(launches) == 2 * (1 + 3)  # RK2: the network once a stage, then the sweeps
    # the corrections do not fit (the sixth allocation of set_learned)
    lean, windows = _run(fake, -1, 5)
    assert whole - lean == 3 * 16 * 4 * NC
    # nor do the FP32 primitives (the first allocation of the block)
    least, same = _run(fake, 0, -1)
    assert lean - least == 8 * 4 * NC
    assert windows == same
    # per stage and direction three windows of 3/8 of the cells each (the lines
    # and their ends are fewer than the cells with ghosts), network and sweep in turn
    assert len(windows) == 2 * 3 * 3 * 2
    assert all(("correct" in a) and ("sweep" in b) for a, b in zip(windows[::2], windows[1::2]))


def test_learned_box_without_any_room_is_refused(fake):
    ig = fake.ig
    for n in range(5):
        blk = ig.GpuBlock(3, N, order="learned")
        fake.fail_in(n)
        with pytest.raises(ig.IdefixError):
            blk.set_learned(np.zeros(NPARAM, np.float32))
        fake.fail_in(-1)
        blk.close()
        assert fake.live_bytes() == 0
