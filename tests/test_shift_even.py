"""GPU: fftShift in place where x and y are even, by pairs of cells (rows of a
multiple of 4, 16-byte aligned images) and by cells, against the reference's
swap loops (ImageFilter.cpp:231-280), which are disjoint there: rolls."""
import numpy as np
import pytest


def _rolled(img, dim, size):
    # the loops leave the last plane (row in 2D) of an odd count alone
    sx, sy, sz = size if dim == 3 else (size[0], 1, size[1])
    a = img.reshape(sz, sy, sx).copy()
    h = sz // 2
    a[:2 * h] = np.roll(a[:2 * h], (h, sy // 2, sx // 2), (0, 1, 2))
    return a.reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])  # cells into a 16-byte aligned buffer
@pytest.mark.parametrize("dim,size,channels", [
    (2, (4, 2, 1), 1), (2, (8, 7, 1), 3), (2, (64, 64, 1), 5), (2, (516, 514, 1), 2), (2, (2, 2, 1), 2),
    (2, (6, 5, 1), 3), (2, (130, 130, 1), 7), (2, (1022, 1023, 1), 3),
    (3, (4, 2, 2), 2), (3, (8, 6, 5), 3), (3, (64, 64, 64), 2), (3, (2, 4, 3), 4), (3, (30, 32, 34), 3), (3, (128, 128, 128), 3)])
def test_shift_even(dim, size, channels, offset):
    import ctypes as C

    import torch

    import fastrecon_gb300 as fr
    rng = np.random.default_rng(5)
    cells = size[0] * size[1] * size[2]
    x = (rng.standard_normal((channels, cells)) + 1j * rng.standard_normal((channels, cells))).astype(np.complex64)
    buf = torch.zeros(channels * cells + 2, dtype=torch.complex64, device="cuda")
    xd = buf[offset:offset + channels * cells]
    xd.copy_(torch.from_numpy(x.ravel()).cuda())
    fr.capi.check(fr.load().fr_fft_shift(C.c_void_p(xd.data_ptr()), channels, dim, fr.capi.u3(size), None), "fr_fft_shift")
    got = xd.cpu().numpy().reshape(channels, cells)
    for c in range(channels):
        assert np.array_equal(got[c], _rolled(x[c], dim, size))
    assert not buf[:offset].any() and not buf[offset + channels * cells:].any()
