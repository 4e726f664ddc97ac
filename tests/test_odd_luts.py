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


@pytest.mark.gpu
@pytest.mark.parametrize("lut_length", LENGTHS)
@pytest.mark.parametrize("dim,G,shape", [(2, 64, (96, 64)), (3, 24, (300, 32))])
def test_gridding_kernels(oracle, dim, G, shape, lut_length):
    """Scatter from tap lists, a batch, Pipe-Menon and a streaming update."""
    import torch

    import fastrecon_gb300 as fr
    from fastrecon_gb300 import batch as fb
    width, coils = 4.0, 7
    traj = synth.golden_angle_2d(*shape) if dim == 2 else synth.kooshball_3d(*shape)
    n = traj.shape[0]
    rng = np.random.default_rng(lut_length)
    kd = (rng.standard_normal((coils, n)) + 1j * rng.standard_normal((coils, n))).astype(np.complex64)
    dcf = rng.uniform(0.2, 1.0, n).astype(np.float32)
    lut = oracle.kb_lut(width, 1.5, lut_length)
    tn = oracle.normalize_traj(traj, dim, G)[0]
    want = oracle.grid_f64(tn, dcf, kd, dim, G, width, lut)
    kt, dt, tt = torch.from_numpy(kd).cuda(), torch.from_numpy(dcf).cuda(), torch.from_numpy(traj).cuda()
    for coil_group in (4, 8, 16):
        plan = fr.GridPlan(dim, G, width, lut=lut, coil_group=coil_group)
        plan.set_trajectory(tt)
        assert plan.tap_words() > 0
        grid = plan.grid(kt, dt)
        assert rel_l2(grid.cpu().numpy(), want) <= TOL
    b = fb.GridBatch(dim, G, width, lut=lut)
    b.set_trajectories(tt, [n])
    assert rel_l2(b.grid(kt.flatten(), dt, coils).cpu().numpy()[0], want) <= TOL
    assert rel_l2(plan.dcf_pipe(3).cpu().numpy(), oracle.dcf_pipe_f64(tn, dim, G, width, lut, 3)) <= 2 * TOL
    new = kd[:, 5:105] * np.float32(1.5)
    plan.update(kt, torch.from_numpy(new).cuda(), 5, dt, grid)
    kd[:, 5:105] = new
    assert rel_l2(grid.cpu().numpy(), oracle.grid_f64(tn, dcf, kd, dim, G, width, lut)) <= TOL
