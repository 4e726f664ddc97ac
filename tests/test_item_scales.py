"""GPU: the per-item fixed-point scales (one block per work item, the first 512
records' bounds kept in registers), over item lengths around that, against the
64-bit reference; samples of zero weight and one far above the others."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("chunk", [1, 33, 128, 511, 512, 513, 1500, 5000])
@pytest.mark.parametrize("dim,coils", [(2, 5), (3, 3), (3, 12)])
def test_scales(oracle, chunk, dim, coils):
    import fastrecon_gb300 as fr
    import torch
    rng = np.random.default_rng(chunk)
    n, G, W = 6000 if chunk > 1 else 300, 40, 4.0
    traj = np.zeros((n, 4), np.float32)
    traj[:, :dim] = rng.uniform(-0.5, 0.5, (n, dim)) * rng.uniform(0, 1, (n, 1)) ** 2
    traj[0, :dim], traj[1, :dim] = -0.5, 0.5
    dcf = rng.uniform(0.5, 1.5, n).astype(np.float32)
    dcf[rng.integers(0, n, n // 10)] = 0.0
    # one sign: no cancellation, so the error is relative to the sums themselves
    kd = (rng.uniform(0.5, 1, (coils, n)) + 1j * rng.uniform(0.5, 1, (coils, n))).astype(np.complex64)
    p = fr.GridPlan(dim, G, W, chunk=chunk)
    p.set_trajectory(torch.from_numpy(traj).cuda())
    assert p.tap_words() > 0
    norm = oracle.normalize_traj(traj, dim, G)[0]
    for peak in (1.0, 1000.0):
        dcf[n // 2] = peak
        got = p.grid(torch.from_numpy(kd).cuda(), torch.from_numpy(dcf).cuda()).cpu().numpy()
        want = oracle.grid_f64(norm, dcf, kd, dim, G, W, p.lut)
        # products to 2^-24 and to 2^-22 of their item's largest, and up to 6000 partial sums of
        # split tiles to 2^-24 each in float
        tol = 5e-7 + (6000 ** 0.5 * 2.0 ** -24 if chunk < 128 else 0)
        if peak > 1:
            # the items that hold the peak (2^dim tiles) round every product to half of 2 peak 2^-22
            taps = 2 ** dim * min(chunk, n) * (13 if dim == 2 else 34)
            tol += (taps * 2 * coils / 12) ** 0.5 * 2 * peak * 2.0 ** -22 / np.linalg.norm(want)
        assert np.linalg.norm(got - want) / np.linalg.norm(want) <= tol
