"""The training step's fused kernels (output layer with the transposed copies,
column sums, gradients + Adam + packed weights) at batch sizes around their
blocks and splits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch_of(n, seed):
    import torch

    g = torch.Generator().manual_seed(seed)
    x = torch.zeros((n, 64), dtype=torch.bfloat16)
    x[:, :30] = torch.randn((n, 30), generator=g)
    return x.cuda(), (torch.rand(n, generator=g) < 0.3).float().cuda()


@pytest.mark.parametrize("batch", [128, 256, 2048, 8192, 16384])
def test_gradients_are_the_mean_over_128_row_batches(batch):
    """dZ is scaled by 1 / batch, a power of two, so its rounding to bf16 is
    that of the 128-row batches and only the order of FP32 sums differs: at
    most 16384 additions of 2^-24 each, 1e-3 of the sum of magnitudes; 1e-4 of
    the gradient's norm leaves room for their random signs."""
    import torch

    from bgt import mlp

    net = mlp.SurvivalMLP(max_batch=16384, seed=7)
    x, y = batch_of(batch, batch)
    g, loss = net.gradients(x, y)
    again, _ = net.gradients(x, y)
    assert torch.equal(g, again)
    parts = [net.gradients(x[s:s + 128].contiguous(), y[s:s + 128].contiguous()) for s in range(0, batch, 128)]
    mean = torch.stack([p[0].double() for p in parts]).mean(0)
    for a, b in ((0, 16384), (16384, 16640), (16640, 82176), (82176, 82432), (82432, 147968), (147968, 148224),
                 (148224, 148480), (148480, 148481)):
        assert torch.linalg.norm(g[a:b].double() - mean[a:b]) <= 1e-4 * torch.linalg.norm(mean[a:b]), (a, b)
    assert abs(loss - np.mean([p[1] for p in parts])) <= 1e-4 * loss


@pytest.mark.parametrize("batch", [128, 9600])
def test_train_step_is_adam_on_the_gradients(batch):
    """Three steps: Adam in FP32 numpy, operation by operation, and the packed
    weights those of a network set to the updated parameters."""
    import torch

    from bgt import mlp

    net = mlp.SurvivalMLP(max_batch=9600, seed=3)
    x, y = batch_of(batch, 1)
    p = net.get_params()
    m, v = np.zeros_like(p), np.zeros_like(p)
    f = np.float32
    b1, b2, lr = f(0.9), f(0.999), f(2e-3)
    for t in range(1, 4):
        g = net.gradients(x, y)[0].cpu().numpy()
        net.train_step(x, y, float(lr))
        m = b1 * m + (f(1) - b1) * g
        v = b2 * v + (f(1) - b2) * g * g
        bc1, bc2 = f(1) - f(float(b1) ** t), f(1) - f(float(b2) ** t)
        p = p - lr * (m / bc1) / (np.sqrt(v / bc2) + f(1e-8))
        assert np.array_equal(net.get_params(), p), t
    other = mlp.SurvivalMLP(max_batch=9600, seed=4)
    other.set_params(p)
    assert torch.equal(net.forward(x[:128].contiguous()), other.forward(x[:128].contiguous()))
    assert torch.equal(net.gradients(x, y)[0], other.gradients(x, y)[0])
