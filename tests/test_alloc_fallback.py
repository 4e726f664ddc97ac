"""GPU: an allocation that fails and is done without leaves no error behind for
the next launch: plans and batches whose tap lists do not fit evaluate the
taps (FR_FAIL_ALLOC_BYTES: reservations of that many bytes or more fail in
cudaMalloc)."""
import numpy as np
import pytest

from conftest import load_case, rel_l2

TOL = 1e-5


@pytest.fixture
def refuse(monkeypatch):
    def at(nbytes):
        monkeypatch.setenv("FR_FAIL_ALLOC_BYTES", str(nbytes))
    return at


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["radial2d_small", "koosh3d_small"])
def test_plan_without_tap_lists(name, refuse):
    import torch

    import fastrecon_gb300 as fr
    c = load_case(name)
    n = c["traj"].shape[0]

    def grid():
        p = fr.GridPlan(c["dim"], c["G"], c["W"], lut=c["lut"], chunk=16384)
        p.set_trajectory(torch.from_numpy(c["traj"]).cuda())
        return p, p.grid(torch.from_numpy(c["kdata"]).cuda(), torch.from_numpy(c["dcf"]).cuda()).cpu().numpy()

    p, _ = grid()
    refuse(n * p.tap_words() * 4)  # the tap slots, the plan's largest reservation
    p, got = grid()
    assert p.tap_words() == 0
    assert rel_l2(got, c["grid"]) <= TOL


@pytest.mark.gpu
def test_batch_without_tap_lists(oracle, refuse):
    import torch

    from fastrecon_gb300 import batch as fb
    c = load_case("radial2d_small")
    n, frames = c["traj"].shape[0], 3
    b = fb.GridBatch(2, c["G"], c["W"], lut=c["lut"], chunk=16384)
    # the batch's tap slots and not one frame's, nor any other buffer
    refuse(frames * n * 12 * 4)
    b.set_trajectories(torch.from_numpy(np.concatenate([c["traj"]] * frames)).cuda(), [n] * frames)
    kd = torch.from_numpy(np.concatenate([c["kdata"].ravel()] * frames)).cuda()
    got = b.grid(kd, torch.from_numpy(np.concatenate([c["dcf"]] * frames)).cuda(), c["kdata"].shape[0]).cpu().numpy()
    assert all(rel_l2(got[f], c["grid"]) <= TOL for f in range(frames))
