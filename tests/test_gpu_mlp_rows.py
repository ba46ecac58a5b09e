"""Classifier inputs at row counts around the feature kernel's blocks, raw and
normalised outputs alone and together, against the same formulas in numpy
(FP64, rounded to FP32 and bf16 at the kernel's points)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 257, 1000])
@pytest.mark.parametrize("raw,normalized", [(True, True), (True, False), (False, True)])
def test_features_row_counts(n, raw, normalized):
    import torch

    from bgt import mlp

    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(n)
    table = rng.standard_normal((2, mlp.VARIANT_COLS)) * 1e-3
    table[:, 10:14] = [[11.9, -1.8, 3.7, 0.47]] * 2
    var = np.sort(rng.integers(0, 2, n)).astype(np.int32)
    v0, v1 = rng.standard_normal((2, 6, n)) * 1e-3
    net = mlp.SurvivalMLP(max_batch=128)
    mean, std = rng.standard_normal(30) * 1e-3, rng.random(30) + 0.5
    net.set_normalization(mean, std)
    x, r = net.features(*(torch.tensor(a, device=dev) for a in (v0, v1, var, table)), raw=raw, normalized=normalized)
    T = table[var]
    f = np.zeros((n, 30))
    f[:, 0:6], f[:, 6:22], f[:, 22:28] = v0.T - T[:, :6], T[:, 14:30], v1.T - T[:, :6]
    dp = f[:, 27]
    xb, pxb, yb, pyb = (f[:, 22 + k] - T[:, 6 + k] * dp for k in range(4))
    ba, aa, bb, ab = T[:, 10:14].T
    f[:, 28] = np.sqrt(0.5 * ((1 + aa * aa) / ba * xb * xb + 2 * aa * xb * pxb + ba * pxb * pxb))
    f[:, 29] = np.sqrt(0.5 * ((1 + ab * ab) / bb * yb * yb + 2 * ab * yb * pyb + bb * pyb * pyb))
    f32 = f.astype(np.float32)
    assert (r is not None) == raw and (x is not None) == normalized
    if raw:
        assert np.array_equal(r.cpu().numpy(), f32)
    if normalized:
        want = np.zeros((mlp.pad_rows(n), 64), np.float32)
        want[:n, :30] = (f32 - mean.astype(np.float32)) * (1.0 / std).astype(np.float32)
        assert torch.equal(x.cpu(), torch.tensor(want).to(torch.bfloat16))


@pytest.mark.parametrize("tiles", [1, 2, 147, 148, 149, 295, 296, 297, 593])
def test_forward_does_not_depend_on_the_tile_schedule(tiles):
    """Rows of a call over `tiles` 128-row tiles (one or two in flight per CTA,
    an odd one left over, several rounds) equal the same rows alone."""
    import torch

    from bgt import mlp

    net = mlp.SurvivalMLP(max_batch=128, seed=5)
    g = torch.Generator().manual_seed(tiles)
    x = torch.randn((128 * tiles, 64), generator=g).to(torch.bfloat16).cuda()
    p = net.forward(x)
    assert torch.isfinite(p).all() and 0 < p.min() and p.max() < 1
    for t in sorted({0, 1, tiles // 3, tiles // 2, tiles - 2, tiles - 1} & set(range(tiles))):
        assert torch.equal(p[128 * t:128 * (t + 1)], net.forward(x[128 * t:128 * (t + 1)].contiguous())), t
    # against the layers in FP32 with activations rounded to bf16: rounding an activation to the other
    # neighbour moves a logit by at most 2^-8 |a w|, and sums differ by reordering only
    w = torch.from_numpy(net.get_params()).cuda()
    a = x.float()
    for o, cols in ((0, 64), (16640, 256), (82432, 256)):
        W = w[o:o + 256 * cols].view(256, cols).to(torch.bfloat16).float()
        a = torch.relu(a.double() @ W.double().T + w[o + 256 * cols:o + 256 * cols + 256].double()).to(
            torch.bfloat16).float()
    z = a @ w[148224:148480].to(torch.bfloat16).float() + w[148480]
    bound = 2.0 ** -8 * (a.abs() @ w[148224:148480].abs()) * 0.25 * 4  # all four rounding points, slope 1/4
    assert ((torch.sigmoid(z) - p).abs() <= bound + 1e-6).all()
