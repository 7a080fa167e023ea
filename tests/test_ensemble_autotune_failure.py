"""An ensemble whose autotuner runs out of memory goes on as before: the same
kernels on the same work lists and segments, by launches and by graph (the
host code on a stand-in for the CUDA runtime)."""
import pytest

from fake_gpu import Fake


@pytest.fixture
def fake(tmp_path, monkeypatch):
    return Fake(tmp_path, monkeypatch)


def _boxes(dims, sizes, precision):
    return [dict(dims=dims, n=(s,) * dims, precision=precision, first_dt=1e-4) for s in sizes]


def _cycle(fake, ens, graph):
    fake.launches()
    ens.run(max_cycles=1, graph=graph)
    return fake.launches()


# 2-D: thread-per-cell sweeps; 3-D of more than 400000 cells: those along x,
# marches along y and z; FP64: nothing to tune, so nothing to fail
@pytest.mark.parametrize("dims,sizes,precision", [(2, (40, 24, 40), "mixed"), (3, (76, 12), "mixed"),
                                                  (2, (40, 24), "fp64")])
def test_failed_autotune_leaves_the_ensemble_as_it_was(fake, dims, sizes, precision):
    ig = fake.ig
    ens = ig.Ensemble(_boxes(dims, sizes, precision))
    before = [_cycle(fake, ens, g) for g in (False, True)]
    segs = [ens.segments(b) for b in range(len(sizes))]
    sweeps = [line for line in before[0] if "ke_sweep" in line]
    assert len(sweeps) == 2 * dims and all(" list " in line for line in sweeps)
    assert before[0] == before[1]
    failed = 0
    for n in range(200):
        fake.fail_in(n)
        try:
            ens.autotune(1)
        except ig.IdefixError:
            failed += 1
        else:
            break
        finally:
            fake.fail_in(-1)
        assert [ens.segments(b) for b in range(len(sizes))] == segs, n
        assert [_cycle(fake, ens, g) for g in (False, True)] == before, n
    assert failed > 10 if precision == "mixed" else failed == 0
    # and the one that had the memory it asked for works on lists that exist
    after = [_cycle(fake, ens, g) for g in (False, True)]
    assert after[0] == after[1] and not any("gone" in line for line in after[0])
