"""The closure's training pass at the edges of its 128-point tiles and of its
grid (296 persistent CTAs): the smallest batch, partial tiles, a batch whose
last CTAs take a second tile and one whose tiles end inside a wave.  Loss and
gradients against the oracle's restatement with the same bf16 roundings, at
the tolerances of test_gpu_closure.py (1e-4 on the loss, 1e-2 on a gradient:
the hardware tanh's 2^-11 through three layers, summed over few points)."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [16, 112, 128, 144, 296 * 128 + 16, 2 * 296 * 128 - 48])
def test_training_gradients_at_tile_edges(h3, orc, P):
    closure = importlib.import_module("3dhit_b200.closure")
    m = closure.ClosureMLP("cuda", seed=P % 97)
    g = torch.Generator().manual_seed(P)
    x = torch.randn(P, 9, generator=g) * 1.5
    tau = torch.randn(P, 6, generator=g) * 0.5
    loss = float(m.loss_and_grads(x.cuda(), tau.cuda()).item())
    m.check_errors()
    _, lo, go = orc.mlp_loss_grads([t.detach().cpu().numpy() for t in m.params], x.numpy(), tau.numpy())
    assert abs(loss - lo) <= 1e-4 * lo
    for p, ref in zip(m.params, go):
        got = p.grad.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(got - ref) <= 1e-2 * np.linalg.norm(ref)
