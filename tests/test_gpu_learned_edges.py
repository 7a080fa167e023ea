"""The learned order's correction launch and cell sweeps (csrc/learned.cu) where
their tiling can go wrong: boxes whose tiles of 128 cells wrap lines and layers
or end early, lines around a sweep's tile, and the wide columns of uct_hll and
uct_hlld.  A network whose outputs are zero, and one whose trained range holds
nothing, leave plain PLM bit for bit, with the right counts of evaluated and
fallen-back cells."""
import os
import sys

import numpy as np
import pytest

import idefix_gb300 as ig
from test_gpu_sweep_cell import _state

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,emf", [((2, 3, 2), "uct_contact"), ((17, 5, 9), "uct_hll"), ((31, 4, 33), "uct_hlld"),
                                   ((62, 7, 3), "arithmetic"), ((6, 126, 5), "uct_contact")])
def test_learned_without_effect_is_plm(n, emf):
    Vc, Vs = _state(n, 5 + sum(n), 2)
    kw = dict(solver="hlld", emf=emf, nstages=2, cfl=0.3, first_dt=1e-4)
    plain = ig.GpuBlock(3, n, order="plm", **kw)
    plain.upload(Vc, Vs)
    plain.run(max_cycles=3)
    ref, t = plain.download(), plain.get_time()
    plain.close()
    for scale, lo, hi in ((0.0, None, None), (1.0, np.ones(216, np.float32), -np.ones(216, np.float32))):
        blk = ig.GpuBlock(3, n, order="learned", **kw)
        blk.set_learned(mlp.init_params(7, out_scale=scale).astype(np.float32), lo, hi)
        blk.upload(Vc, Vs)
        blk.run(max_cycles=3)
        out = blk.download()
        assert blk.get_time() == t
        assert np.array_equal(out[0], ref[0]) and np.array_equal(out[1], ref[1])
        cells, fell = blk.learned_stats()
        assert cells > 0 and fell == (cells if lo is not None else 0)
        blk.close()
