"""The training step's blocks of 128 samples (csrc/train_tile.cuh) where they
can go wrong: batches that end before, at and after a block, a feature array
without 16-byte alignment, the range of the features the training saw, and
repeated runs, which agree bit for bit (nothing in a step depends on timing).
Gradients against the float64 oracle with the same bfloat16 rounding of weights
and layer inputs: relative L2 error below 2e-2 (bfloat16 keeps 8 bits)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 2e-2


@pytest.fixture(scope="module", autouse=True)
def built():
    from idefix_gb300 import build

    build.build_library()


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, dtype=np.float64) - b) / max(np.linalg.norm(b), 1e-300))


def _batch(B, seed=3):
    rng = np.random.default_rng(seed)
    X = torch.zeros((B, 224), dtype=torch.float32)
    X[:, :216] = torch.from_numpy(0.3 * rng.standard_normal((B, 216))).float()
    T = torch.from_numpy(0.1 * rng.standard_normal((B, 16))).float()
    return X.to(torch.bfloat16).cuda().contiguous(), T.cuda().contiguous()


def _dataset(S=2, nc=9, seed=1):
    g = torch.Generator().manual_seed(seed)
    P = 0.2 * torch.randn((S, 8, nc, nc, nc), generator=g)
    P[:, (0, 4)] = 1.0 + 0.3 * torch.rand((S, 2, nc, nc, nc), generator=g)
    return P.cuda().contiguous(), torch.rand((S, 3, 16, nc**3), generator=g).cuda().contiguous()


@pytest.mark.parametrize("B", [1, 31, 127, 128, 129, 257, 640])
def test_gradients_at_block_edges(B):
    from idefix_gb300 import learned

    params = mlp.init_params(3, out_scale=0.5).astype(np.float32)
    X, T = _batch(B)
    tr = learned.Trainer(max_batch=640, params=params)
    g, loss = tr.grad(X, T)
    Xq = X.float().cpu().numpy()[:, :216].astype(np.float64)
    l0, g0 = mlp.loss_and_grad(params.astype(np.float64), Xq, T.cpu().numpy().astype(np.float64), quant=True)
    assert abs(loss - l0) < TOL * l0
    G, G0 = mlp.unpack(g), mlp.unpack(g0)
    for k in ("W1", "b1", "W2", "b2", "W3", "b3"):
        assert _rel(G[k], G0[k]) < TOL, k
    Y0, _ = mlp.forward(params.astype(np.float64), Xq, quant=True)
    assert _rel(tr.forward(X).cpu().numpy(), Y0) < TOL
    # the same batch from an array that starts between 16-byte boundaries
    Xs = torch.empty(B * 224 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(B, 224)
    Xs.copy_(X)
    torch.cuda.synchronize()
    assert Xs.data_ptr() % 16 == 2
    g2, loss2 = tr.grad(Xs, T)
    assert np.array_equal(g, g2) and loss == loss2


@pytest.mark.parametrize("B,steps", [(1, 2), (128, 1), (200, 3), (512, 5)])
def test_training_repeats_and_sees_its_features(B, steps):
    from idefix_gb300 import learned

    P, T = _dataset()
    torch.cuda.synchronize()
    params = mlp.init_params(4, out_scale=0.1).astype(np.float32)
    runs = []
    for _ in range(2):
        tr = learned.Trainer(max_batch=512, params=params)
        tr.set_dataset(P, T)
        losses = tr.train(steps, B, lr=1e-3, lr_end=1e-4, seed=9)
        runs.append((losses, tr.get_params(), *tr.feature_range()))
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    # the range is that of the batches' features (which the batch call rounds to bfloat16)
    X = torch.cat([tr.batch(B, seed=9, base=s * B)[0] for s in range(steps)]).float().cpu().numpy()[:, :216]
    for got, want in ((runs[0][2], X.min(0)), (runs[0][3], X.max(0))):
        assert np.all(np.abs(got - want) <= 2.0**-8 * np.abs(want) + 1e-30)
    # the first step's loss is that batch's loss before any update
    X0, T0 = tr.batch(B, seed=9, base=0)
    torch.cuda.synchronize()
    _, loss = learned.Trainer(max_batch=512, params=params).grad(X0, T0)
    assert abs(runs[0][0][0] - loss) <= 1e-6 * loss
