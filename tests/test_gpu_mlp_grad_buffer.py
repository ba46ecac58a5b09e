"""bgt_mlp_gradients into a caller's array: one that the kernel can write
itself, and one that is not aligned to a float, which only a copy can."""
from __future__ import annotations

import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4, 1, 2, 3])
def test_gradients_reach_any_array(offset):
    import torch

    from bgt import mlp

    net = mlp.SurvivalMLP(max_batch=256, seed=3)
    g = torch.Generator().manual_seed(1)
    x = torch.zeros((256, 64), dtype=torch.bfloat16)
    x[:, :30] = torch.randn((256, 30), generator=g)
    x, y = x.cuda(), (torch.rand(256, generator=g) < 0.3).float().cuda()
    want, loss = net.gradients(x, y)
    raw = torch.full((4 * mlp.N_PARAMS + 8,), 255, dtype=torch.uint8, device="cuda")
    got = C.c_float()
    rc = net.lib.bgt_mlp_gradients(net.h, x.data_ptr(), y.data_ptr(), 256, raw.data_ptr() + offset, C.byref(got),
                                   torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and abs(got.value - loss) <= 8 * 2.0 ** -24 * loss  # four sums added in any order
    torch.cuda.synchronize()
    assert torch.equal(raw[offset:offset + 4 * mlp.N_PARAMS], want.view(torch.uint8))
    rest = torch.cat([raw[:offset], raw[offset + 4 * mlp.N_PARAMS:]])
    assert bool((rest == 255).all())
