"""Batches through the tap lists: every frame equals the reference algorithm's
grid, for frames of no, one and many samples, several coil groups and tilings
(tap lanes of 8 and 16 warps, and the kernel that evaluates the taps), direct
and replayed."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5


def _frames(dim):
    if dim == 2:
        return [synth.spiral_2d(3, 700), synth.golden_angle_2d(1, 1), synth.radial_2d(31, 77), synth.spiral_2d(9, 512)]
    return [synth.kooshball_3d(90, 24), synth.kooshball_3d(31, 17), synth.kooshball_3d(200, 32)]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,width,tile,chunk,coil_group,coils,checkerboard", [
    (2, 48, 4.0, (0, 0, 0), 0, 0, 12, False), (2, 48, 4.0, (32, 16, 0), 256, 16, 17, True),
    (2, 33, 4.0, (16, 16, 0), 512, 8, 3, False), (2, 48, 5.0, (0, 0, 0), 0, 4, 6, False),
    (2, 48, 4.0, (64, 32, 0), 0, 8, 5, False),     # too large for the tap lanes
    (2, 48, 4.0, (16, 16, 0), 0, 32, 20, False),   # coil groups of 32
    (2, 48, 4.0, (0, 0, 0), 0, 0, 1, True),
    (3, 24, 4.0, (0, 0, 0), 0, 0, 16, True), (3, 21, 3.0, (8, 4, 4), 256, 8, 9, False),
    (3, 20, 5.0, (8, 8, 8), 0, 16, 4, False),      # no tap lists
])
def test_batch_frames(oracle, dim, G, width, tile, chunk, coil_group, coils, checkerboard):
    import torch

    from fastrecon_gb300 import batch as fb
    trajs = _frames(dim)
    trajs[1][0] = 0 if trajs[1].shape[0] > 1 else trajs[1][0]
    rng = np.random.default_rng(G + coils)
    dcfs = [rng.uniform(0.2, 1.0, t.shape[0]).astype(np.float32) for t in trajs]
    kds = [(rng.standard_normal((coils, t.shape[0])) + 1j * rng.standard_normal((coils, t.shape[0]))).astype(np.complex64)
           for t in trajs]
    use = [i for i, t in enumerate(trajs) if t.shape[0] > 1]  # one sample has no range to normalise with
    trajs, dcfs, kds = ([x[i] for i in use] for x in (trajs, dcfs, kds))
    counts = [t.shape[0] for t in trajs]
    counts.insert(1, 0)  # an empty frame
    lut = oracle.kb_lut(width, 1.5, 512)
    b = fb.GridBatch(dim, G, width, lut=lut, tile=tile, chunk=chunk, coil_group=coil_group, checkerboard=checkerboard)
    b.set_trajectories(torch.from_numpy(np.concatenate(trajs)).cuda(), counts)
    kd = torch.from_numpy(np.concatenate([k.ravel() for k in kds])).cuda()
    dcf = torch.from_numpy(np.concatenate(dcfs)).cuda()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        rep = b.capture(kd, dcf, coils, stream=s)
        got = b.grid(kd, dcf, coils, stream=s)
        b.replay(stream=s)
    torch.cuda.synchronize()
    sign = np.where(np.indices((G,) * dim).sum(0).ravel() % 2, -1.0, 1.0) if checkerboard else 1.0
    assert not got[1].any()
    for out in (got.cpu().numpy(), rep.cpu().numpy()):
        for f, (t, d, k) in zip([0] + list(range(2, len(counts))), zip(trajs, dcfs, kds)):
            tn = oracle.normalize_traj(t, dim, G)[0]
            want = oracle.grid(tn, d, k, dim, G, width, lut, threads=4) * sign
            assert rel_l2(out[f], want) <= TOL


@pytest.mark.gpu
def test_batch_weak_and_broken_coils(oracle):
    """A coil 10^6 times weaker than the others is gridded as well as by the
    kernel that evaluates the taps with a scale per coil (coil groups of 32),
    and a coil with an infinity leaves the others as they were."""
    import torch

    from fastrecon_gb300 import batch as fb
    t = synth.radial_2d(61, 64)
    rng = np.random.default_rng(5)
    k = (rng.standard_normal((5, t.shape[0])) + 1j * rng.standard_normal((5, t.shape[0]))).astype(np.complex64)
    k[2] *= np.float32(1e-6)
    dcf = rng.uniform(0.2, 1.0, t.shape[0]).astype(np.float32)
    lut = oracle.kb_lut(4.0, 2.0, 512)
    want = oracle.grid_f64(oracle.normalize_traj(t, 2, 64)[0], dcf, k, 2, 64, 4.0, lut)

    def grid(kd, **kw):
        b = fb.GridBatch(2, 64, 4.0, lut=lut, **kw)
        b.set_trajectories(torch.from_numpy(t).cuda(), [t.shape[0]])
        return b.grid(torch.from_numpy(kd.ravel()).cuda(), torch.from_numpy(dcf).cuda(), 5).cpu().numpy()[0]

    got, each = grid(k), grid(k, coil_group=32, tile=(16, 16, 0))
    # two bits of the fixed-point step: a coil's largest value is scaled to [1, 2),
    # and an item's scale serves its largest coil
    bound = [4 * rel_l2(each[c], want[c]) for c in range(5)]
    assert all(rel_l2(got[c], want[c]) <= bound[c] for c in range(5))
    k[1, 100] = np.inf
    bad = grid(k)
    assert all(rel_l2(bad[c], want[c]) <= bound[c] for c in (0, 2, 3, 4))


@pytest.mark.gpu
def test_batch_quiet_runs(oracle):
    """A coil that is all but silent in every fourth run of 128 samples, the
    first among them, is gridded like the others."""
    import torch

    from fastrecon_gb300 import batch as fb
    t = synth.radial_2d(32, 64)
    rng = np.random.default_rng(6)
    k = (rng.standard_normal((3, t.shape[0])) + 1j * rng.standard_normal((3, t.shape[0]))).astype(np.complex64)
    k[1, (np.arange(t.shape[0]) // 128) % 4 == 0] *= np.float32(1e-37)
    dcf = rng.uniform(0.2, 1.0, t.shape[0]).astype(np.float32)
    lut = oracle.kb_lut(4.0, 2.0, 512)
    b = fb.GridBatch(2, 64, 4.0, lut=lut)
    b.set_trajectories(torch.from_numpy(t).cuda(), [t.shape[0]])
    got = b.grid(torch.from_numpy(k.ravel()).cuda(), torch.from_numpy(dcf).cuda(), 3).cpu().numpy()[0]
    want = oracle.grid(oracle.normalize_traj(t, 2, 64)[0], dcf, k, 2, 64, 4.0, lut, threads=4)
    assert all(rel_l2(got[c], want[c]) <= TOL for c in range(3))
