"""The kernel's mass summed by LUT entries equals the midpoint sum over radii."""
import numpy as np
import pytest

from fastrecon_gb300.learned_dcf import kernel_mass


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("width,length,steps", [
    (4.0, 512, 100000), (3.0, 512, 100000), (5.5, 333, 100000), (4.0, 2, 100000), (4.0, 1, 1000), (2.7, 4096, 1000),
    (4.0, 51, 100), (4.0, 101, 100), (12.9, 1024, 100000), (4.0, 512, 511),
])
def test_kernel_mass(dim, width, length, steps):
    lut = np.random.default_rng(length).uniform(0, 1, length).astype(np.float32)
    hw = width / 2
    r = (np.arange(steps) + 0.5) * (hw / steps)
    k = lut.astype(np.float64)[np.minimum(np.rint(r / hw * (length - 1)).astype(np.int64), length - 1)]
    want = np.sum(k * (2 * np.pi * r if dim == 2 else 4 * np.pi * r * r)) * (hw / steps)
    # both sums in 64 bits, all terms positive: a few roundings each
    assert abs(kernel_mass(lut, width, dim, steps) - want) <= 1e-13 * want
