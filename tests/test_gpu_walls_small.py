"""The boundary pass of boxes about as small as their ghost layers (one launch
per direction where every ghost's image is an active cell, two where it is not)
and mixed-precision runs with walls, whose stage begins fill the ghosts alone:
every value of both whole arrays against the oracle, ghosts included; the mixed
run against the same run with a fresh start of the run before every cycle."""
import numpy as np
import pytest

import idefix_gb300 as ig
from mhd_state import extract
from test_gpu_sweep_cell import _state

pytestmark = pytest.mark.gpu
O, R, PER = ("outflow", "outflow"), ("reflective", "reflective"), ("periodic", "periodic")


@pytest.mark.parametrize("n,order,bc", [
    ((2, 5), "ppm", (O, R)), ((2, 2), "plm", (R, R)), ((3, 4), "ppm", (R, ("outflow", "reflective"))),
    ((2, 3, 2), "ppm", (O, O, O)), ((3, 2, 4), "plm", (PER, R, O)), ((4, 3, 3), "ppm", (R, R, R)),
])
def test_boundary_pass_of_small_boxes_matches_oracle(n, order, bc):
    from oracle.pyofx import Oracle

    D = len(n)
    blk, o = ig.GpuBlock(D, n, order=order, bc=bc), Oracle(D, n, order=order, bc=bc)
    rng = np.random.default_rng(8)
    Vc, Vs = rng.standard_normal(blk.vc_shape), rng.standard_normal(blk.vs_shape)
    blk.upload(Vc, Vs)
    o.set_prim(Vc, Vs)
    blk.set_boundaries()
    o.lib.ofx_set_boundaries(o.h)
    got, want = blk.download(), o.get_prim()
    blk.close()
    assert np.array_equal(got[0][:2 * D + 2], want[0][:2 * D + 2])
    assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("n,stages,bc", [((40, 31), 2, (O, R)), ((23, 34), 3, (O, PER)), ((12, 10, 14), 2, (R, O, PER))])
def test_mixed_runs_with_walls_do_not_depend_on_their_pieces(n, stages, bc):
    D = len(n)
    Vc, Vs = _state(n, 3, 2)
    out = []
    for pieces in ((5,), (1, 1, 1, 1, 1)):
        blk = ig.GpuBlock(D, n, precision="mixed", nstages=stages, cfl=0.3, first_dt=1e-4, bc=bc)
        blk.upload(Vc, Vs)
        for c in pieces:
            blk.run(max_cycles=c)
        out.append((extract(D, n, 2, *blk.download()), blk.get_time()))
        blk.close()
    (a, ta), (b, tb) = out
    assert ta == tb
    assert np.array_equal(a[0], b[0])
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)
