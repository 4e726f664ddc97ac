"""GPU: the 2D transform at every number of columns per block (16 for one coil,
8 for two and where 4 would take two rounds of blocks, else 4), and its x stage by
blocks of lines and by warps, against a 64-bit transform."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("G", [240, 320, 384, 640])
@pytest.mark.parametrize("coils,out", [(1, (0, -1)), (1, (-100, 0)), (2, (0, 0)), (2, (-3, -30)), (2, (-4, -4)), (3, (0, 0)),
                                       (5, (0, -8)), (8, (-8, 0)), (20, (-120, -2))])
def test_plane_columns(G, coils, out):
    import torch

    import fastrecon_gb300 as fr
    rx, ry = G + out[0], G + out[1]
    rng = np.random.default_rng(G + coils)
    g = (rng.standard_normal((coils, G, G)) + 1j * rng.standard_normal((coils, G, G))).astype(np.complex64)
    got = fr.gridding.CropSoS(2, G, coils, (rx, ry, 1))(torch.from_numpy(g).cuda()).cpu().numpy().reshape(ry, rx)
    x0, y0 = (G - rx) // 2, (G - ry) // 2
    img = np.fft.ifft2(g.astype(np.complex128), axes=(1, 2), norm="forward")[:, y0:y0 + ry, x0:x0 + rx]
    want = np.sqrt((np.abs(img) ** 2).sum(0))
    # log2(G^2) < 19 roundings of 2^-24 each on the way at most add up to 1.2e-6, in the mean far less
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-6
