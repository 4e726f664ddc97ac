"""GPU: the 3D transform's x stage by blocks of lines (most outputs kept, no tile
mask) and by warps, against a 64-bit transform."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("G", [240, 256])
@pytest.mark.parametrize("rx", [1.0, 0.61, 0.59])
def test_volume(G, rx):
    import torch

    import fastrecon_gb300 as fr
    R = (int(rx * G), 32, 20)
    rng = np.random.default_rng(G)
    g = (rng.standard_normal((1, G, G, G)) + 1j * rng.standard_normal((1, G, G, G))).astype(np.complex64)
    got = fr.gridding.CropSoS(3, G, 1, R)(torch.from_numpy(g).cuda()).cpu().numpy().reshape(R[::-1])
    sl = [slice((G - r) // 2, (G - r) // 2 + r) for r in R[::-1]]
    a = g[0].astype(np.complex128)
    for axis in range(3):
        a = np.fft.ifft(a, axis=axis, norm="forward")[tuple(sl[axis] if k == axis else slice(None) for k in range(3))]
    want = np.abs(a)
    # log2(G^3) = 24 roundings of 2^-24 each on the way at most add up to 1.5e-6, in the mean far less
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-6
