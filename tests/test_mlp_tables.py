"""GPU: the network's inference reads the same tables from parameters that are not
16-byte aligned."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [1, 2, 4, 7])
def test_unaligned_parameters(offset):
    import torch

    from fastrecon_gb300 import learned_dcf as ld
    net = ld.DCFNet(seed=3)
    x = torch.from_numpy(np.random.default_rng(0).standard_normal((777, 5)).astype(np.float32)).cuda()
    want = net.forward(x).clone()
    buf = torch.empty(ld.N_PARAMS + 8, dtype=torch.bfloat16, device="cuda")
    net.bf16 = buf[offset:offset + ld.N_PARAMS].copy_(net.bf16)
    assert torch.equal(net.forward(x), want)
