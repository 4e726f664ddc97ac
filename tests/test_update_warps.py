"""Incremental regridding at coil counts around a warp, wide footprints and
single samples: the updated grid and k-space against a full regrid by the
FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5  # the project's gridding bar


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,width,coils,begin,count", [
    (2, 32, 4.0, 1, 7, 1), (2, 33, 6.0, 31, 0, 40), (2, 32, 3.0, 32, 100, 33), (3, 16, 4.0, 33, 64, 100),
    (3, 18, 5.0, 5, 10, 257), (3, 20, 7.0, 2, 3, 9)])
def test_update_matches_regrid(oracle, dim, G, width, coils, begin, count):
    import torch

    import fastrecon_gb300 as fr
    traj = synth.golden_angle_2d(20, 30) if dim == 2 else synth.kooshball_3d(40, 16)
    n = traj.shape[0]
    rng = np.random.default_rng(coils)
    kd = (rng.standard_normal((coils, n)) + 1j * rng.standard_normal((coils, n))).astype(np.complex64)
    new = (rng.standard_normal((coils, count)) + 1j * rng.standard_normal((coils, count))).astype(np.complex64)
    dcf = rng.uniform(0.1, 1.0, n).astype(np.float32)
    lut = oracle.kb_lut(width, 1.5, 512)
    plan = fr.GridPlan(dim, G, width, lut=lut)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    kdev, ddev = torch.from_numpy(kd).cuda(), torch.from_numpy(dcf).cuda()
    grid = plan.grid(kdev, ddev)
    plan.update(kdev, torch.from_numpy(new).cuda(), begin, ddev, grid)
    kd[:, begin:begin + count] = new
    assert np.array_equal(kdev.cpu().numpy(), kd)
    tn = oracle.normalize_traj(traj, dim, G)[0]
    assert rel_l2(grid.cpu().numpy(), oracle.grid_f64(tn, dcf, kd, dim, G, width, lut)) <= TOL
