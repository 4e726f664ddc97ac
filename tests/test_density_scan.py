"""Density counts where the one-pass plane scan, the per-cell histogram's slots
and the clamped boxes meet their edges: exact against the oracle."""
import numpy as np
import pytest

from fastrecon_gb300 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,shape", [(2, 31, (40, 50)), (2, 64, (300, 200)), (3, 5, (30, 16)), (3, 31, (200, 32)),
                                         (3, 33, (200, 40)), (3, 67, (300, 64)), (3, 96, (900, 96))])
def test_counts_exact(oracle, dim, G, shape):
    import torch

    import fastrecon_gb300 as fr
    from fastrecon_gb300 import learned_dcf as ld
    traj = synth.golden_angle_2d(*shape) if dim == 2 else synth.kooshball_3d(*shape)
    traj[:, 1] *= 1.2  # some samples are clamped to the border cells
    plan = fr.GridPlan(dim, G, 4.0)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    got = ld.density_counts(plan).cpu().numpy()
    tn = oracle.normalize_traj(traj, dim, G)[0]
    assert np.array_equal(got, oracle.density_counts(tn, dim, G, list(ld.RADII)))


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,n", [(3, 40, 2), (3, 40, 17), (3, 67, 4097), (2, 64, 1001)])
@pytest.mark.parametrize("radii", [(3,), (0, 1, 5), (1, 2, 4, 8, 16), (0, 1, 2, 3, 7, 30, 63, 100)])
def test_counts_radii(oracle, dim, G, n, radii):
    """Numbers of radii around the four at a time, boxes from a cell to the whole grid, odd sample counts."""
    import torch

    import fastrecon_gb300 as fr
    from fastrecon_gb300 import learned_dcf as ld
    traj = np.zeros((n, 4), np.float32)
    traj[:, :dim] = np.random.default_rng(n).uniform(-0.5, 0.5, (n, dim)) * ([1, 1.2, 1][:dim])
    plan = fr.GridPlan(dim, G, 4.0)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    tn = oracle.normalize_traj(traj, dim, G)[0]
    got = ld.density_counts(plan, radii).cpu().numpy()
    assert np.array_equal(got, oracle.density_counts(tn, dim, G, list(radii)))
