"""GPU: a reconstruction after one that filled the whole grid: the transform's
lines without samples, whose cells the gridding leaves unwritten, are zero and
not what the other reconstruction left there."""
import numpy as np
import pytest

from fastrecon_gb300 import synth


@pytest.mark.gpu
@pytest.mark.parametrize("G,out,tile,coils,squeeze", [
    (64, (42, 42, 42), (0, 0, 0), 3, (1, 1, 1)), (64, (48, 48, 48), (16, 8, 4), 9, (1, 0.3, 0.6)),
    (64, (45, 46, 47), (8, 4, 16), 2, (1, 0.2, 1)), (128, (96, 96, 96), (4, 4, 4), 1, (1, 0.05, 0.5)),
    (160, (112, 80, 100), (8, 8, 8), 2, (1, 1, 0.1)), (192, (128, 128, 128), (0, 0, 0), 1, (1, 0.5, 1)),
])
def test_lines_left_out(G, out, tile, coils, squeeze):
    import torch

    import fastrecon_gb300 as fr
    rng = np.random.default_rng(G + coils)
    full = np.zeros((4 * G * G, 4), np.float32)
    full[:, :3] = rng.uniform(-0.5, 0.5, (4 * G * G, 3))
    ball = synth.kooshball_3d(300, G).copy()
    ball[:, :3] *= np.asarray(squeeze, np.float32)
    recon = G * 2 // 3 if G % 3 == 0 else G // 2
    os = 1.5 if G % 3 == 0 else 2.0

    def make(**kw):
        return fr.Recon(3, recon, os, coils, out_size=out, tile=tile, deterministic=True, **kw)

    def run(rec, traj, seed):
        r = np.random.default_rng(seed)
        n = traj.shape[0]
        k = (r.standard_normal((coils, n)) + 1j * r.standard_normal((coils, n))).astype(np.complex64)
        dcf = r.uniform(0.2, 1.0, n).astype(np.float32)
        return rec.run(*(torch.from_numpy(a).cuda() for a in (traj, dcf, k))).cpu().numpy()

    kept = make(pruned_fft=True)
    run(kept, full, 1)
    got = run(kept, ball, 2)
    assert np.array_equal(got, run(make(pruned_fft=True), ball, 2))
    want = run(make(use_cufft=True), ball, 2).astype(np.float64)
    # two transforms of log2(G^3) < 23 roundings of 2^-24 on the way each
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2.8e-6
