"""GPU: the tap-lane scatter of at most 8 coils (rows of 2 or 4 copies of a
cell, added up at the flush) and of large tiles, against the per-warp tap
lists (the same fixed-point sums: equal bits) and the reference algorithm."""
import os

import numpy as np
import pytest

from conftest import load_case, rel_l2

TOL = 1e-5


def _grid(torch, c, kd, **kw):
    import fastrecon_gb300 as fr
    p = fr.GridPlan(c["dim"], c["G"], c["W"], lut=c["lut"], deterministic=True, **kw)
    p.set_trajectory(torch.from_numpy(c["traj"]).cuda())
    assert p.tap_words() > 0
    return p.grid(torch.from_numpy(kd).cuda(), torch.from_numpy(c["dcf"]).cuda()).cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["radial2d_small", "radial2d_oddgrid", "koosh3d_small", "koosh3d_odd"])
@pytest.mark.parametrize("coil_group,coils", [(4, 1), (4, 4), (4, 7), (8, 5), (8, 8), (8, 11), (16, 2), (16, 7), (16, 12)])
@pytest.mark.parametrize("tile,chunk,checkerboard", [((0, 0, 0), 0, True), ((8, 4, 4), 512, False), ((6, 8, 2), 0, False)])
def test_few_coils_equal_warp_lists(oracle, name, coil_group, coils, tile, chunk, checkerboard):
    import torch
    c = load_case(name)
    if tile[0] % (32 // min(2 * coil_group, 32)):
        pytest.skip("the plan refuses this tile for this coil group")
    checkerboard = checkerboard and c["G"] % 2 == 0
    rng = np.random.default_rng(coils)
    n = c["traj"].shape[0]
    kd = (rng.standard_normal((coils, n)) + 1j * rng.standard_normal((coils, n))).astype(np.complex64)
    kw = dict(coil_group=coil_group, tile=tile, chunk=chunk, checkerboard=checkerboard)
    got = _grid(torch, c, kd, **kw)
    os.environ["FR_SCATTER_WARP_LISTS"] = "1"
    try:
        lists = _grid(torch, c, kd, **kw)
    finally:
        os.environ.pop("FR_SCATTER_WARP_LISTS", None)
    assert np.array_equal(got.view(np.uint32), lists.view(np.uint32))
    if not checkerboard:
        want = oracle.grid(c["traj_norm"], c["dcf"], kd, c["dim"], c["G"], c["W"], c["lut"], threads=4)
        assert rel_l2(got, want) <= TOL
