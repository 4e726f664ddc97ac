"""GPU: an allocation that fails and is done without leaves no error behind for
the next launch: plans and batches whose tap lists do not fit evaluate the
taps (FR_FAIL_ALLOC_BYTES: reservations of that many bytes or more fail in
cudaMalloc), and whatever memory a batch without tap lists can be planned and
gridded in is enough for the same batch with them (FR_ALLOC_LIMIT_BYTES: the
reservations held may not exceed that)."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [0, 256])
def test_batch_within_any_limit(chunk, monkeypatch):
    import gc

    import torch

    import fastrecon_gb300 as fr
    from fastrecon_gb300 import batch as fb
    from fastrecon_gb300.capi import FastreconError
    c = load_case("radial2d_small")
    n, frames, coils = c["traj"].shape[0], 6, c["kdata"].shape[0]
    traj = torch.from_numpy(np.concatenate([c["traj"]] * frames)).cuda()
    kd = torch.from_numpy(np.concatenate([c["kdata"].ravel()] * frames)).cuda()
    dcf = torch.from_numpy(np.concatenate([c["dcf"]] * frames)).cuda()

    def run(limit, lists):
        gc.collect()
        monkeypatch.delenv("FR_ALLOC_LIMIT_BYTES", raising=False)
        b = fb.GridBatch(2, c["G"], c["W"], lut=c["lut"], chunk=chunk, tap_lists=lists)
        monkeypatch.setenv("FR_ALLOC_LIMIT_BYTES", str(limit))
        try:
            for _ in range(2):  # planned again over the buffers of the first time
                b.set_trajectories(traj, [n] * frames)
                before = fr.kernel_launches()
                got = b.grid(kd, dcf, coils).cpu().numpy()
                launches = fr.kernel_launches() - before
        except FastreconError as e:
            assert e.status == 3
            return None
        assert all(rel_l2(got[f], c["grid"]) <= TOL for f in range(frames))
        return launches

    seen = set()
    for limit in np.geomspace(2e5, 2e7, 60).astype(int):
        plain, lists = run(limit, False), run(limit, True)
        assert (plain is None) == (lists is None) or plain is None, limit
        seen.add((plain, lists))
    assert (None, None) in seen
    kinds = {b for a, b in seen if a is not None}
    assert len(kinds) == 2  # with and without the lists
