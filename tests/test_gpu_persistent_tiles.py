"""The persistent ensemble launch's FP64 sweeps (tiles of 64 cells, csrc/
sweep_cell.cuh) at box sizes around a tile: lines that end before, at and after
one, totals that leave a tile of a cell or two, boxes smaller than one.  Every
box evolves as the same box run alone, bit for bit."""
import numpy as np
import pytest

import idefix_gb300 as ig
from test_gpu_sweep_cell import _state

pytestmark = pytest.mark.gpu

SIZES2 = [(2, 2), (3, 2), (2, 31), (58, 3), (60, 2), (61, 5), (62, 3), (63, 2), (29, 30), (30, 62), (124, 7)]
SIZES3 = [(2, 3, 2), (60, 2, 3), (61, 4, 2), (3, 30, 5), (5, 2, 62)]


@pytest.mark.parametrize("sizes,order", [(SIZES2, "plm"), (SIZES2, "ppm"), (SIZES3, "plm"), (SIZES3, "ppm")])
def test_persistent_sweeps_at_tile_edges(sizes, order):
    ng = 3 if order == "ppm" else 2
    kws = [dict(dims=len(n), n=n, order=order, cfl=0.3, first_dt=1e-4) for n in sizes]
    states = [_state(n, 11 + k, ng) for k, n in enumerate(sizes)]
    ens = ig.Ensemble(kws)
    for k, s in enumerate(states):
        ens.upload(k, *s)
    ens.run(max_cycles=4, persistent=True)
    for k, (kw, s) in enumerate(zip(kws, states)):
        blk = ig.GpuBlock(kw["dims"], kw["n"], **{q: kw[q] for q in ("order", "cfl", "first_dt")})
        blk.upload(*s)
        blk.run(max_cycles=4)
        a, b = ens.download(k), blk.download()
        g = ng
        act = (slice(None),) + tuple(slice(g, g + n) if n > 1 else slice(None)
                                     for n in reversed(list(kw["n"]) + [1] * (3 - kw["dims"])))
        assert np.array_equal(a[0][act], b[0][act]), sizes[k]
        for c in range(kw["dims"]):
            fx = tuple(slice(g, g + n + (1 if d == c else 0)) if d < kw["dims"] else slice(None)
                       for d, n in reversed(list(enumerate(list(kw["n"]) + [1] * (3 - kw["dims"])))))
            assert np.array_equal(a[1][c][fx], b[1][c][fx]), (sizes[k], c)
        assert ens.get_time(k)[:3] == blk.get_time(), sizes[k]
        blk.close()
    ens.close()
