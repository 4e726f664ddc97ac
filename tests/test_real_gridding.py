"""Real-valued gridding from the tap lists and the degridding of the Pipe-Menon
iteration, at the sizes where tiles, kernel footprints and split tiles meet
grid edges, against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL_GRID = 1e-5  # FP32 sums of up to a few thousand terms vs FP64
TOL_PIPE = 2e-5  # 3 iterations: each adds the rounding of one gridding and one degridding

CASES = [  # dim, G, width, tile, chunk, (spokes, readout)
    (2, 64, 4.0, (0, 0, 0), 0, (96, 64)),
    (2, 61, 4.0, (12, 20, 0), 300, (64, 96)),     # tiles that are no powers of two, an odd grid
    (2, 40, 5.0, (8, 8, 0), 0, (40, 60)),         # footprint as wide as a tile's half
    (2, 33, 3.0, (32, 32, 0), 512, (50, 40)),     # a last tile of one cell
    (2, 48, 7.5, (16, 8, 0), 0, (48, 48)),        # up to 8 cells along x
    (3, 24, 4.0, (0, 0, 0), 256, (300, 32)),
    (3, 21, 3.0, (8, 4, 12), 0, (200, 24)),
    (3, 20, 5.0, (8, 8, 8), 0, (150, 24)),        # no tap lists (more than 60 taps a sample)
]


def _plan(oracle, dim, G, width, tile, chunk, traj, **kw):
    import torch

    import fastrecon_gb300 as fr
    lut = oracle.kb_lut(width, 1.5, 512)
    plan = fr.GridPlan(dim, G, width, lut=lut, tile=tile, chunk=chunk, **kw)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    return plan, lut


def _traj(dim, shape):
    return synth.golden_angle_2d(*shape) if dim == 2 else synth.kooshball_3d(*shape)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,width,tile,chunk,shape", CASES)
def test_real_gridding_and_pipe(oracle, dim, G, width, tile, chunk, shape):
    import torch
    traj = _traj(dim, shape)
    plan, lut = _plan(oracle, dim, G, width, tile, chunk, traj)
    tn = oracle.normalize_traj(traj, dim, G)[0]
    w = np.random.default_rng(1).uniform(0.1, 1.0, traj.shape[0]).astype(np.float32)
    got = plan.grid_real(torch.from_numpy(w).cuda()).cpu().numpy()
    want = oracle.grid_real_f64(tn, w.astype(np.float64), dim, G, width, lut)
    assert rel_l2(got, want) <= TOL_GRID
    assert np.array_equal(got == 0, want == 0)
    got = plan.dcf_pipe(3).cpu().numpy()
    assert rel_l2(got, oracle.dcf_pipe_f64(tn, dim, G, width, lut, 3)) <= TOL_PIPE


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_real_gridding_keeps_non_finite_weights(oracle, bad):
    """An infinite or NaN weight reaches exactly the cells it reaches when
    each record's box is evaluated."""
    import torch
    traj = _traj(3, (60, 24))
    w = np.ones(traj.shape[0], np.float32)
    w[777] = bad
    out = [_plan(oracle, 3, 24, 4.0, (0, 0, 0), 0, traj, tap_lists=t)[0].grid_real(torch.from_numpy(w).cuda())
           .cpu().numpy() for t in (True, False)]
    assert np.array_equal(np.isfinite(out[0]), np.isfinite(out[1]))
    assert (~np.isfinite(out[0])).any()


@pytest.mark.gpu
def test_pipe_with_few_samples_per_tile(oracle):
    traj = _traj(3, (6, 16))
    plan, lut = _plan(oracle, 3, 64, 4.0, (0, 0, 0), 0, traj)
    tn = oracle.normalize_traj(traj, 3, 64)[0]
    assert rel_l2(plan.dcf_pipe(3).cpu().numpy(), oracle.dcf_pipe_f64(tn, 3, 64, 4.0, lut, 3)) <= TOL_PIPE
