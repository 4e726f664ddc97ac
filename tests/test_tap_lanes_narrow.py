"""GPU: the tap-lane scatter of at most 4 coils (rows of 4 copies of a cell) on
tiles of up to 512 cells, which plans with coil groups of 8 and 16 take there (those
of 4 take the per-warp lists), against the lists and the reference algorithm."""
import numpy as np
import pytest

from conftest import load_case, rel_l2

TOL = 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["radial2d_small", "radial2d_oddgrid", "koosh3d_small", "koosh3d_odd"])
@pytest.mark.parametrize("coil_group,coils", [(8, 1), (8, 3), (8, 4), (16, 1), (16, 4)])
@pytest.mark.parametrize("tile,chunk", [((8, 8, 8), 0), ((8, 4, 4), 512), ((6, 8, 2), 0)])
def test_narrow_lanes(oracle, monkeypatch, name, coil_group, coils, tile, chunk):
    import torch

    import fastrecon_gb300 as fr
    c = load_case(name)
    if tile[0] % (32 // min(2 * coil_group, 32)):
        pytest.skip("the plan refuses this tile for this coil group")
    rng = np.random.default_rng(coils)
    n = c["traj"].shape[0]
    kd = (rng.standard_normal((coils, n)) + 1j * rng.standard_normal((coils, n))).astype(np.complex64)
    got = []
    for lists in ("0", "1"):
        monkeypatch.setenv("FR_SCATTER_WARP_LISTS", lists)
        p = fr.GridPlan(c["dim"], c["G"], c["W"], lut=c["lut"], deterministic=True, coil_group=coil_group, tile=tile,
                        chunk=chunk)
        p.set_trajectory(torch.from_numpy(c["traj"]).cuda())
        assert p.tap_words() > 0
        got.append(p.grid(torch.from_numpy(kd).cuda(), torch.from_numpy(c["dcf"]).cuda()).cpu().numpy())
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    want = oracle.grid(c["traj_norm"], c["dcf"], kd, c["dim"], c["G"], c["W"], c["lut"], threads=4)
    assert rel_l2(got[0], want) <= TOL
