"""The FP64 flux sweeps with one thread per cell (csrc/sweep_cell.cuh) where
their tiling can go wrong: lines that end just before, at and after the end of
a tile of 32, 64 or 128 positions (two of them shared with the next tile,
three with PPM; two columns side by side across x), an odd number of columns,
the smallest boxes, and boxes large enough for the largest block.  Every active
cell, evolved face and the time step equal the oracle's bit for bit."""
import numpy as np
import pytest

import idefix_gb300 as ig
from mhd_state import embed, extract
from oracle.pyofx import Oracle

pytestmark = pytest.mark.gpu


def _state(n, seed, ng):
    """smooth random box of any size (edge-centred vector potential, so div B = 0)"""
    D = len(n)
    rng = np.random.default_rng(seed)
    m = list(n) + [1] * (3 - D)
    shape = (m[2], m[1], m[0])
    noise = lambda: rng.standard_normal(shape)  # noqa: E731
    vc = np.zeros((2 * D + 2,) + shape)
    vc[0] = 1.0 + 0.2 * np.tanh(noise())
    for d in range(D):
        vc[1 + d] = 0.3 * np.tanh(noise())
    vc[D + 1] = 0.6 + 0.1 * np.tanh(noise())
    A = [0.02 * noise() for _ in range(3)]
    dif = lambda a, d: (np.roll(a, -1, axis=2 - d) - a) * m[d] if d < D else 0.0  # noqa: E731
    B = [dif(A[2], 1) - dif(A[1], 2), dif(A[0], 2) - dif(A[2], 0), dif(A[1], 0) - dif(A[0], 1)]
    scale = 0.3 / max(np.abs(b).max() for b in B[:D])
    vs = []
    for d in range(D):
        b = 0.1 + scale * B[d]
        vs.append(np.concatenate([b, np.take(b, [0], axis=2 - d)], axis=2 - d))
    return embed(D, n, ng, vc, vs)


CASES = [  # (n, order, solver, emf, stages)
    ((2, 2), "plm", "hlld", "uct_contact", 2),
    ((3, 2), "ppm", "hlld", "uct_contact", 2),
    ((28, 30), "plm", "hlld", "uct_contact", 2),
    ((60, 61), "plm", "hlld", "uct_contact", 2),
    ((62, 63), "limo3", "hlld", "uct_hll", 2),
    ((64, 59), "ppm", "roe", "uct_contact", 3),
    ((126, 125), "order1", "hll", "arithmetic", 1),
    ((127, 124), "ppm", "hlld", "uct_hlld", 2),
    ((128, 500), "plm", "tvdlf", "uct0", 2),
    ((2, 3, 2), "plm", "hlld", "uct_contact", 2),
    ((5, 2, 61), "limo3", "hlld", "uct_contact", 2),
    ((59, 62, 3), "ppm", "hlld", "uct_contact", 2),
    ((31, 29, 30), "plm", "roe", "uct_hlld", 3),
    ((63, 64, 65), "plm", "hlld", "uct_contact", 2),
    ((66, 33, 40), "ppm", "hll", "uct_hll", 2),
]


@pytest.mark.parametrize("n,order,solver,emf,stages", CASES)
def test_cell_sweeps_match_oracle_at_tile_edges(n, order, solver, emf, stages):
    D = len(n)
    ng = 3 if order == "ppm" else 2
    Vc, Vs = _state(n, 17 + sum(n), ng)
    kw = dict(order=order, solver=solver, emf=emf, nstages=stages, cfl=0.3, first_dt=1e-4)
    blk = ig.GpuBlock(D, n, **kw)
    blk.upload(Vc, Vs)
    blk.run(max_cycles=3)
    got, t = extract(D, n, ng, *blk.download()), blk.get_time()
    blk.close()
    o = Oracle(D, n, **kw)
    o.set_prim(Vc, Vs)
    assert o.run(max_cycles=3) == 0
    want = extract(D, n, ng, *o.get_prim())
    assert t == o.get_time()
    assert np.array_equal(got[0], want[0])
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)
