"""The FP32 flux sweeps with one thread per cell (csrc/sweep_cell.cuh, the mixed
path's small boxes) against the marching sweeps, which the ensemble's persistent
launch runs at every size: the same arithmetic, so equal bits.  Sizes around the
end of a tile's line (126 positions along x, 14 across it in blocks of 128, 62
and 30 in smaller ones), the smallest boxes, and boxes on either side of the sizes where the sweeps
change form."""
import numpy as np
import pytest

import idefix_gb300 as ig
from mhd_state import extract
from test_gpu_sweep_cell import _state

pytestmark = pytest.mark.gpu

CASES = [  # (n, order, solver, emf, stages)
    ((2, 2), "plm", "hlld", "uct_contact", 2),
    ((3, 2), "ppm", "hlld", "uct_contact", 2),
    ((29, 31), "plm", "hlld", "uct_contact", 2),
    ((61, 13), "limo3", "hlld", "uct_hll", 2),
    ((125, 127), "ppm", "roe", "uct_contact", 3),
    ((126, 14), "order1", "hll", "arithmetic", 1),
    ((500, 311), "plm", "tvdlf", "uct0", 2),
    ((1030, 1024), "plm", "hlld", "uct_contact", 2),  # y: marches on both sides
    ((2, 3, 2), "plm", "hlld", "uct_contact", 2),
    ((13, 15, 61), "limo3", "hlld", "uct_contact", 2),
    ((59, 12, 3), "ppm", "hlld", "uct_hlld", 2),
    ((33, 28, 30), "plm", "roe", "uct_hlld", 3),
    ((66, 33, 40), "ppm", "hll", "uct_hll", 2),
    ((76, 74, 72), "plm", "hlld", "uct_contact", 2),  # y, z: marches
    ((176, 162, 150), "plm", "hlld", "uct_contact", 2),  # x: warp chunks
]


@pytest.mark.parametrize("n,order,solver,emf,stages", CASES)
def test_cell_sweeps_match_marches(n, order, solver, emf, stages):
    D = len(n)
    ng = 3 if order == "ppm" else 2
    Vc, Vs = _state(n, 23 + sum(n), ng)
    kw = dict(order=order, solver=solver, emf=emf, nstages=stages, cfl=0.3, first_dt=1e-4, precision="mixed")
    blk = ig.GpuBlock(D, n, **kw)
    blk.upload(Vc, Vs)
    blk.run(max_cycles=3)
    a, ta = extract(D, n, ng, *blk.download()), blk.get_time()
    blk.close()
    for persistent in (True, False):
        ens = ig.Ensemble([dict(dims=D, n=n, **kw)])
        ens.upload(0, Vc, Vs)
        ens.run(max_cycles=3, persistent=persistent)
        b, tb = extract(D, n, ng, *ens.download(0)), ens.get_time(0)
        ens.close()
        assert tuple(ta)[:3] == tuple(tb)[:3]
        assert np.array_equal(a[0], b[0])
        for x, y in zip(a[1], b[1]):
            assert np.array_equal(x, y)
