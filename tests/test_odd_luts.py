"""GPU: kernels that stage the kernel table in shared memory, for tables of an
odd number of entries (whatever follows such a table has to be aligned by
itself)."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5  # FP32 sums of up to 125 taps vs FP64

LENGTHS = [3, 333, 511, 1023]


@pytest.mark.gpu
@pytest.mark.parametrize("lut_length", LENGTHS)
@pytest.mark.parametrize("dim,G,width,shape,coils", [
    (2, 182, 4.0, (400, 256), 12), (2, 190, 5.0, (400, 260), 32), (3, 36, 4.0, (1800, 50), 12), (3, 35, 4.0, (14000, 50), 6),
])
def test_degrid_tiles(oracle, dim, G, width, shape, coils, lut_length):
    import torch

    import fastrecon_gb300 as fr
    traj = synth.golden_angle_2d(*shape) if dim == 2 else synth.kooshball_3d(*shape)
    lut = oracle.kb_lut(width, 1.5, lut_length)
    plan = fr.GridPlan(dim, G, width, lut=lut)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    rng = np.random.default_rng(G + lut_length)
    g = (rng.standard_normal((coils, G ** dim)) + 1j * rng.standard_normal((coils, G ** dim))).astype(np.complex64)
    before = fr.kernel_launches()
    got = plan.degrid(torch.from_numpy(g).cuda()).cpu().numpy()
    assert fr.kernel_launches() - before == 2  # the tiled form
    tn = oracle.normalize_traj(traj, dim, G)[0]
    want = oracle.degrid_f64(tn, g.astype(np.complex128), dim, G, width, lut)
    assert rel_l2(got, want) <= TOL
