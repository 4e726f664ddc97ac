"""The training step's gradient at the edges of its 64-sample tiles and beyond
one tile per CTA, against the FP64 oracle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 30001])
def test_gradient_at_tile_edges(oracle, n):
    import torch

    from fastrecon_gb300 import learned_dcf as ld
    rng = np.random.default_rng(n)
    net = ld.DCFNet(seed=3)
    x = rng.uniform(-4, 4, (n, ld.N_IN)).astype(np.float32)
    t = rng.uniform(-6, 2, n).astype(np.float32)
    c = rng.uniform(0, 2, n).astype(np.float32)
    loss = float(net.loss_grad(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), torch.from_numpy(c).cuda()))
    first = net.grad.cpu().numpy().copy()
    lw, gw = oracle.mlp_backward(net.params_bf16_as_float(), x, t, c)
    assert abs(loss - lw) <= 1e-5 * abs(lw)
    assert np.linalg.norm(first - gw) <= 1e-5 * np.linalg.norm(gw)  # FP32 sums of up to 30,001 terms, tile by tile
    net.loss_grad(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), torch.from_numpy(c).cuda())
    assert np.array_equal(first, net.grad.cpu().numpy())  # fixed order
