"""HLLD on states it has no solution for: with a negative density beside the
face a star state's root is a NaN, and the flux of the double-star region is one
in every variable, the density and the normal momentum included.  One stage
against the CPU oracle, values and places
of the NaNs."""
import numpy as np
import pytest

import idefix_gb300 as ig
from idefix_gb300 import ic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from idefix_gb300 import build

    build.build_library()
    build.build_oracle()


@pytest.mark.parametrize("dims,n", [(2, (32, 28)), (3, (16, 12, 10))])
def test_stage_with_negative_densities_matches_oracle(dims, n):
    from oracle.pyofx import Oracle

    g = 2
    Vc, Vs = ic.turbulence_3d(16, seed=5, kmax=4) if dims == 3 else ic.orszag_tang_2d(32)
    m = tuple(n) + (1,) * (3 - dims)
    nt = [m[d] + 2 * g if d < dims else 1 for d in range(3)]
    fx = [x + 1 if d < dims else 1 for d, x in enumerate(nt)]
    Vc = np.ascontiguousarray(Vc[:, :nt[2], :nt[1], :nt[0]])
    Vs = np.ascontiguousarray(Vs[:, :fx[2], :fx[1], :fx[0]])
    rng = np.random.default_rng(8)
    act = (slice(g, g + m[2]) if dims == 3 else slice(None), slice(g, g + m[1]), slice(g, g + m[0]))
    rho = Vc[0][act]
    bad = rng.random(rho.shape) < 0.05
    rho[bad] *= -0.3 - rng.random(int(bad.sum()))
    blk, o = ig.GpuBlock(dims, n), Oracle(dims, n)
    blk.upload(Vc, Vs)
    o.set_prim(Vc, Vs)
    blk.set_boundaries()
    o.lib.ofx_set_boundaries(o.h)
    blk.prim_to_cons()
    o.lib.ofx_prim_to_cons(o.h)
    blk.reset_stage()
    o.lib.ofx_reset_stage(o.h)
    blk.evolve_stage(0.0, 1e-4)
    o.lib.ofx_evolve_stage(o.h, 0.0, 1e-4)
    got, want = blk.download_cons(), o.get_cons()
    for v in range(2 * dims + 2):
        a, b = got[v][act], want[v][act]
        assert np.array_equal(np.isnan(a), np.isnan(b)), v
        assert np.array_equal(a, b, equal_nan=True), v
    assert np.isnan(want[0][act]).any() and not np.isnan(want[0][act]).all()
    blk.close()
