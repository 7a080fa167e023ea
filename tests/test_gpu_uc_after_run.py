"""What download_cons hands out on the mixed path after a run, whose stage ends
leave the field part of Uc to be rebuilt: the conserved state of the run also
where new arrays have been uploaded since or a further run had nothing to do,
and the state that prim_to_cons made."""
import numpy as np
import pytest

import idefix_gb300 as ig
from test_gpu_sweep_cell import _state

pytestmark = pytest.mark.gpu

WALLS = {2: (("outflow", "reflective"), ("periodic", "periodic")),
         3: (("periodic", "periodic"), ("outflow", "outflow"), ("reflective", "outflow"))}


def _block(n, walls, **kw):
    if walls:
        kw["bc"] = WALLS[len(n)]
    return ig.GpuBlock(len(n), n, precision="mixed", cfl=0.3, first_dt=1e-4, **kw)


def _active(n):
    return (slice(None),) + tuple(slice(2, 2 + m) if m else slice(None) for m in reversed(list(n) + [0] * (3 - len(n))))


@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("n", [(33, 20), (14, 9, 11)])
def test_prim_to_cons_after_a_run(n, walls):
    other = _state(n, 5, 2)
    other[0][len(n) + 2:] += 0.25  # a cell field that is not the mean of the faces
    got = []
    for run in (False, True):
        blk = _block(n, walls)
        if run:
            blk.upload(*_state(n, 4, 2))
            blk.run(max_cycles=2)
        blk.upload(*other)
        blk.prim_to_cons()
        got.append(blk.download_cons()[_active(n)])
        blk.close()
    assert np.array_equal(*got)


@pytest.mark.parametrize("kw", [{}, dict(nstages=1), dict(check_nan_period=2), dict(nstages=3, emf="uct_hll")])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("n", [(33, 20), (14, 9, 11)])
def test_conserved_state_of_a_run(n, walls, kw):
    first, other = _state(n, 4, 2), _state(n, 5, 2)
    got = []
    for later in ("nothing", "upload", "set_boundaries", "no run"):
        blk = _block(n, walls, **kw)
        blk.upload(*first)
        blk.run(max_cycles=3)
        if later in ("upload", "no run"):
            blk.upload(*other)
        if later == "set_boundaries":
            blk.set_boundaries()
        if later == "no run":
            blk.set_time(1.0, 1e-4)
            blk.run(tstop=0.5)  # past its end already
        got.append(blk.download_cons()[_active(n)])
        if later == "nothing":  # and a second time, and against the means of the faces
            assert np.array_equal(blk.download_cons()[_active(n)], got[0])
            vs = blk.download()[1]
            for d in range(len(n)):
                f = vs[d][tuple(slice(2, 2 + m + (a == d)) if m else slice(0, 1)
                                for a, m in reversed(list(enumerate(list(n) + [0] * (3 - len(n))))))]
                ax = 2 - d
                lo, hi = np.take(f, range(f.shape[ax] - 1), axis=ax), np.take(f, range(1, f.shape[ax]), axis=ax)
                assert np.array_equal(got[0][len(n) + 2 + d], 0.5 * (lo + hi))
        blk.close()
    for g in got[1:]:
        assert np.array_equal(g, got[0])
