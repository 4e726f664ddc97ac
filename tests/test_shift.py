"""fftShift in place at every mix of odd and even axes: the swap groups of the
parallel kernel against the reference's swap loops (ImageFilter.cpp:231-280)
replayed one by one."""
import numpy as np
import pytest

SIZES = [(2, (1, 1, 1)), (2, (1, 2, 1)), (2, (2, 3, 1)), (2, (3, 2, 1)), (2, (7, 9, 1)), (2, (33, 64, 1)),
         (3, (1, 1, 2)), (3, (2, 3, 4)), (3, (3, 3, 3)), (3, (3, 4, 5)), (3, (4, 5, 3)), (3, (5, 1, 7)),
         (3, (17, 33, 9)), (3, (32, 7, 18))]


def _replay(img, dim, size):
    sx, sy, sz = size if dim == 3 else (size[0], 1, size[1])
    a = img.reshape(sz, sy, sx).copy()
    hx, hy, hz = sx // 2, sy // 2, sz // 2
    for z in range(hz):
        for y in range(sy):
            y1 = y + hy if y < hy else y - hy
            for x in range(sx):
                x1 = x + hx if x < hx else x - hx
                a[z, y, x], a[z + hz, y1, x1] = a[z + hz, y1, x1], a[z, y, x]
    return a.reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,size", SIZES)
def test_shift_replays_the_swaps(dim, size):
    import ctypes as C

    import torch

    import fastrecon_gb300 as fr
    rng = np.random.default_rng(5)
    cells = size[0] * size[1] * size[2]
    x = (rng.standard_normal((2, cells)) + 1j * rng.standard_normal((2, cells))).astype(np.complex64)
    xd = torch.from_numpy(x).cuda()
    fr.capi.check(fr.load().fr_fft_shift(C.c_void_p(xd.data_ptr()), 2, dim, fr.capi.u3(size), None), "fr_fft_shift")
    got = xd.cpu().numpy()
    for c in range(2):
        assert np.array_equal(got[c], _replay(x[c], dim, size))
