"""Training and evaluation over batches that take a block through more than one
tile of 128 assembled samples (csrc/train_tile.cuh): two (129 to 8192 with an
odd number of 64-sample chunks), three and more (above 16384).  The parameters after one
step against Adam's formula, in float32 as the kernel has it, on the gradients
that grad() gives for the same samples (each operation rounded once: within a
few units of the last place of weight or step), and the losses of eval() against
the network's outputs (float32 outputs, float64 sums: 1e-6)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp  # noqa: E402
from test_gpu_train_tile import _dataset  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
MASKED = (5, 13)  # the normal field: not in the loss


@pytest.mark.parametrize("B", [129, 300, 8192 - 64, 16500])
def test_step_and_losses_over_several_tiles(B):
    from idefix_gb300 import learned

    P, T = _dataset()
    torch.cuda.synchronize()
    params = mlp.init_params(4, out_scale=0.1).astype(np.float32)
    tr = learned.Trainer(max_batch=B, params=params)
    tr.set_dataset(P, T)
    X, Y = tr.batch(B, seed=9, base=0)
    g, loss = tr.grad(X, Y)
    g = np.asarray(g, dtype=np.float32)
    lr = np.float32(1e-3)
    losses = tr.train(1, B, lr=float(lr), lr_end=float(lr), seed=9)
    assert abs(losses[0] - loss) <= 1e-6 * loss
    one = np.float32(1.0)
    b1, b2, eps = np.float32(0.9), np.float32(0.999), np.float32(1e-8)
    m, v = (one - b1) * g, (one - b2) * g * g
    bc1, bc2 = np.float32(1.0 - float(b1)), np.float32(1.0 - float(b2))
    want = params - lr * (m / bc1) / (np.sqrt(v / bc2) + eps)
    got = tr.get_params()
    assert np.all(np.abs(got - want) <= 2.0**-21 * np.maximum(np.abs(params), lr))
    moved = np.abs(got - params) > 0.5 * lr
    assert moved.mean() > 0.5  # (gradients of dead inputs are zero)
    # eval: the samples from base 0 of its seed, without a backward pass
    tr = learned.Trainer(max_batch=B, params=params)
    tr.set_dataset(P, T)
    e, e0 = tr.eval(B, seed=9)
    keep = [o for o in range(16) if o not in MASKED]
    y, t = tr.forward(X).cpu().numpy()[:, keep], Y.cpu().numpy()[:, keep]
    assert abs(e - np.sum((y - t).astype(np.float64) ** 2) / B) <= 1e-6 * e
    assert abs(e0 - np.sum(t.astype(np.float64) ** 2) / B) <= 1e-6 * e0
