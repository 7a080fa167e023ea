"""A learned box on a device that has no room left for the corrections of all
three directions, and on one with none for the FP32 primitives either: the same
states, times and counts, bit for bit, as with all of the memory (the rest of the
device is held by another array meanwhile)."""
import os
import sys

import numpy as np
import pytest

import idefix_gb300 as ig
from test_gpu_sweep_cell import _state

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,emf", [((150, 141, 146), "uct_contact"), ((71, 590, 66), "uct_hlld")])
def test_learned_box_in_windows(n, emf):
    torch = pytest.importorskip("torch")
    Vc, Vs = _state(n, 3, 2)
    params = mlp.init_params(7, out_scale=0.02).astype(np.float32)
    lo, hi = np.full(216, -0.5, np.float32), np.full(216, 0.5, np.float32)
    nc = int(np.prod(Vc.shape[1:]))
    doubles = 46 * nc + 2 * Vs.size + (12 * nc if emf == "uct_hlld" else 0)  # the solver's fields
    # launches of the network per cycle: one a stage, or a window a launch
    windows = sum(-(-((n[a] + 2 * e) * (n[b] + 2 * e)) // ((6 * nc // 16) // (n[d] + 2)))
                  for e in [2 if emf == "uct_hlld" else 1]
                  for d, a, b in ((0, 1, 2), (1, 0, 2), (2, 0, 1)))
    runs = []
    for room in (None, 8 * (doubles + 4 * nc) + 300 * 2**20, 8 * doubles + 60 * 2**20):
        hold = None
        if room:  # 4 nc doubles are the FP32 primitives, 24 nc the corrections
            assert 300 * 2**20 < 8 * 24 * nc and 60 * 2**20 < 8 * 4 * nc
            torch.cuda.empty_cache()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        blk = ig.GpuBlock(3, n, order="learned", emf=emf, cfl=0.3, first_dt=1e-4)
        blk.set_learned(params, lo, hi)
        blk.upload(Vc, Vs)
        blk.profile(True)
        blk.run(max_cycles=2)
        launches = blk.profile_read()["learned_recon"][1]
        blk.profile(False)
        runs.append((*blk.download(), blk.get_time(), blk.learned_stats(), launches))
        blk.close()
        del hold
        torch.cuda.empty_cache()
    a, b, c = runs
    assert a[4] == 2 * 2 and b[4] == c[4] == 2 * 2 * windows
    cells, fell = a[3]
    assert 0 < fell < cells
    for x in (b, c):
        assert np.array_equal(x[0], a[0]) and np.array_equal(x[1], a[1])
        assert x[2:4] == a[2:4]
