"""GPU: the tap lanes with 64-bit indices (tap words past 2^31), for every row
width and for batches, against the scatter that evaluates the taps."""
import pytest

TOL = 1e-5  # the project's gridding bar


def _traj(torch, spokes, readout, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    d = torch.randn((spokes, 3), device="cuda", generator=g)
    d /= d.norm(dim=1, keepdim=True)
    t = torch.zeros((spokes, readout, 4), device="cuda")
    t[:, :, :3] = d[:, None, :] * ((torch.arange(readout, device="cuda") - readout / 2) / readout)[None, :, None]
    return t.reshape(-1, 4)


def _rel(a, b):
    return ((a - b).norm() / b.norm()).item()


@pytest.mark.gpu
@pytest.mark.parametrize("coils,coil_group", [(2, 8), (6, 8), (10, 16)])
def test_plan_past_32_bits(coils, coil_group):
    import torch

    import fastrecon_gb300 as fr
    t = _traj(torch, 200000, 256, 1)
    n = t.shape[0]
    g = torch.Generator(device="cuda").manual_seed(2)
    kd = torch.randn((coils, n), dtype=torch.complex64, device="cuda", generator=g)
    dcf = torch.rand(n, device="cuda", generator=g)
    out = []
    for lists in (True, False):
        p = fr.GridPlan(3, 128, 4.0, coil_group=coil_group, tap_lists=lists)
        p.set_trajectory(t)
        assert not lists or n * p.tap_words() >= 2 ** 31
        out.append(p.grid(kd, dcf))
        del p
    for c in range(coils):
        assert _rel(out[0][c], out[1][c]) <= TOL


@pytest.mark.gpu
def test_batch_past_32_bits():
    import torch

    from fastrecon_gb300 import batch as fb
    t = torch.cat([_traj(torch, 130000, 256, 3), _traj(torch, 70000, 256, 4)])
    counts, coils = [130000 * 256, 70000 * 256], 6
    g = torch.Generator(device="cuda").manual_seed(5)
    kd = torch.randn(coils * t.shape[0], dtype=torch.complex64, device="cuda", generator=g)
    dcf = torch.rand(t.shape[0], device="cuda", generator=g)
    out = []
    for lists in (True, False):
        b = fb.GridBatch(3, 128, 4.0, tap_lists=lists)
        b.set_trajectories(t, counts)
        out.append(b.grid(kd, dcf, coils))
        del b
    for f in range(2):
        for c in range(coils):
            assert _rel(out[0][f, c], out[1][f, c]) <= TOL
