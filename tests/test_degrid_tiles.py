"""Tiled degridding at the edges of tiles, tile parts, coil groups and
footprints, against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5  # FP32 sums of up to 125 taps vs FP64

CASES = [  # dim, G, width, tile, chunk, (spokes, readout), coils, checkerboard, tiled
    (2, 182, 4.0, (0, 0, 0), 0, (400, 256), 12, True, True),
    (2, 183, 4.0, (12, 20, 0), 0, (400, 260), 13, False, True),   # odd grid, tiles that are no powers of two
    (2, 190, 5.0, (8, 64, 0), 0, (400, 260), 32, True, True),     # two groups of coils
    (2, 182, 3.5, (32, 32, 0), 512, (400, 256), 16, False, True),
    (3, 36, 4.0, (0, 0, 0), 512, (1800, 50), 12, False, True),
    (3, 36, 4.0, (0, 0, 0), 0, (1400, 50), 16, True, True),       # parts of 2 planes
    (3, 35, 4.0, (8, 4, 12), 0, (14000, 50), 6, False, True),     # 3 pairs on 4 lanes, under 8 coils
    (3, 33, 4.0, (0, 0, 0), 0, (3000, 50), 8, False, True),       # 4 pairs on 4 lanes
    (3, 33, 3.7, (8, 8, 8), 0, (1100, 50), 32, True, True),       # two groups
    (3, 20, 5.0, (8, 8, 8), 0, (400, 24), 33, True, False),       # a width-5 grid within the cache
    (2, 64, 6.0, (0, 0, 0), 0, (200, 64), 4, False, False),       # footprints over 5 cells
    (3, 64, 4.0, (0, 0, 0), 0, (20, 24), 6, False, False),        # few samples
]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,width,tile,chunk,shape,coils,checkerboard,tiled", CASES)
def test_degrid_tiles(oracle, dim, G, width, tile, chunk, shape, coils, checkerboard, tiled):
    import torch

    import fastrecon_gb300 as fr
    traj = synth.golden_angle_2d(*shape) if dim == 2 else synth.kooshball_3d(*shape)
    traj[:, 1] *= 1.3  # some samples leave the grid along y
    lut = oracle.kb_lut(width, 1.5, 512)
    plan = fr.GridPlan(dim, G, width, lut=lut, tile=tile, chunk=chunk, checkerboard=checkerboard)
    plan.set_trajectory(torch.from_numpy(traj).cuda())
    rng = np.random.default_rng(G)
    g = (rng.standard_normal((coils, G ** dim)) + 1j * rng.standard_normal((coils, G ** dim))).astype(np.complex64)
    out = torch.full((coils, traj.shape[0]), float("nan"), dtype=torch.complex64, device="cuda")
    before = fr.kernel_launches()
    got = plan.degrid(torch.from_numpy(g).cuda(), out=out).cpu().numpy()
    assert fr.kernel_launches() - before == (2 if tiled else 1)  # the tiled form also clears samples off the grid
    gin = g.astype(np.complex128)
    if checkerboard:
        gin = gin * np.where(np.indices((G,) * dim).sum(0).ravel() % 2, -1.0, 1.0)[None]
    tn = oracle.normalize_traj(traj, dim, G)[0]
    want = oracle.degrid_f64(tn, gin, dim, G, width, lut)
    assert np.isfinite(got).all()
    assert np.array_equal(got == 0, want == 0)
    assert rel_l2(got, want) <= TOL
