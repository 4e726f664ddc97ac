"""GPU: the 2D transform with four columns of several coils per block, against a
64-bit transform: coil counts around a block's four, column counts that leave a
block part empty (and odd ones, which skip the staged copies)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("G", [64, 128, 160, 192, 240, 256, 320, 384, 480, 512, 640])
@pytest.mark.parametrize("coils,out", [(1, (0, 0)), (3, (-30, -31)), (4, (-22, -20)), (9, (-27, -2)), (5, (0, -7))])
def test_plane_sos(G, coils, out):
    import fastrecon_gb300 as fr
    import torch
    rx, ry = G + out[0], G + out[1]
    rng = np.random.default_rng(G + coils)
    g = (rng.standard_normal((coils, G, G)) + 1j * rng.standard_normal((coils, G, G))).astype(np.complex64)
    deapod = rng.uniform(0.5, 2.0, (ry, rx)).astype(np.float32) if coils == 3 else None
    got = fr.gridding.CropSoS(2, G, coils, (rx, ry, 1))(
        torch.from_numpy(g).cuda(), deapod=None if deapod is None else torch.from_numpy(deapod).cuda())
    x0, y0 = (G - rx) // 2, (G - ry) // 2
    img = np.fft.ifft2(g.astype(np.complex128), axes=(1, 2), norm="forward")[:, y0:y0 + ry, x0:x0 + rx]
    want = np.sqrt((np.abs(img) ** 2).sum(0))
    if deapod is not None:
        want = want / deapod
    got = got.cpu().numpy().reshape(ry, rx)
    # log2(G^2) < 19 roundings of 2^-24 each on the way at most add up to 1.2e-6, in the mean far less
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-6
