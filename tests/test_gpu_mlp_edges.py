# SPDX-License-Identifier: Apache-2.0
"""The gradient kernel's edges: one row, a full tile, one row more, one tile more than the resident CTAs, and feature rows
off the 16-byte boundaries its wide loads need; each against PyTorch autograd in FP32 with the kernel's BF16 operand
rounding, and the same bits when repeated (every sum has a fixed order)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from alloy_b200.solvers.sph.warmstart import Network, init_params, unpack

pytestmark = pytest.mark.gpu


def _gradient(p, x, t):
    u = {k: torch.tensor(v, dtype=torch.float32, device=x.device, requires_grad=True) for k, v in unpack(p).items()}
    bf = lambda a: a + (a.to(torch.bfloat16).float() - a).detach()  # noqa: E731
    h = bf(x) @ bf(u["w1"]).T + u["b1"]
    h = h * torch.sigmoid(h)
    h = bf(h) @ bf(u["w2"]).T + u["b2"]
    h = h * torch.sigmoid(h)
    loss = ((h @ u["w3"].T + u["b3"] - t) ** 2).sum() / (2 * len(x))
    loss.backward()
    return {k: v.grad for k, v in u.items()}, float(loss.detach())


@pytest.mark.parametrize("batch", [1, 128, 129, 2 * 148 * 128 + 1])
def test_gradient_at_tile_edges(cuda, batch):
    g = torch.Generator(device=cuda).manual_seed(batch)
    rows = torch.randn(16 * (batch + 7) + 1, generator=g, device=cuda)
    t = torch.randn((batch + 7, 2), generator=g, device=cuda)
    idx = torch.randperm(batch + 7, generator=g, device=cuda)[:batch].to(torch.int32)
    x = rows[1:].view(batch + 7, 16)  # 4 bytes off the boundary
    p = init_params(seed=5)
    net = Network(p)
    aligned, loss = net.gradient(x.clone(), t, idx)
    again, _ = net.gradient(x.clone(), t, idx)
    off, loss_off = net.gradient(x, t, idx)
    net.status()
    np.testing.assert_array_equal(aligned, again)
    np.testing.assert_array_equal(aligned, off)
    assert loss == loss_off
    ref, ref_loss = _gradient(p, x[idx.long()], t[idx.long()])
    assert loss == pytest.approx(ref_loss, rel=2e-3)  # the tolerances of test_gpu_mlp.py
    for k, r in unpack(aligned).items():
        want = ref[k].cpu().numpy().reshape(r.shape)
        np.testing.assert_allclose(r, want, rtol=0, atol=2e-2 * float(np.abs(want).max()) + 1e-9, err_msg=k)
