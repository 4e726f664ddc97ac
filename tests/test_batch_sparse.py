"""GPU: batches of sparse frames, on both sides of the line between the tap lanes and
the scatter that evaluates the taps, against the reference algorithm."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5

CASES = [  # dim, G, coils, samples per frame, tap lanes
    (2, 64, 12, 200, False), (2, 64, 12, 400, True), (2, 64, 7, 100, False), (2, 64, 7, 150, True),
    (2, 64, 3, 60, False), (2, 64, 3, 100, True), (3, 24, 12, 200, False), (3, 24, 12, 300, True), (3, 24, 5, 20, True)]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,coils,n,lanes", CASES)
def test_sparse_frames(oracle, dim, G, coils, n, lanes):
    import torch

    import fastrecon_gb300 as fr
    from fastrecon_gb300 import batch as fb
    full = synth.golden_angle_2d(40, 32) if dim == 2 else synth.kooshball_3d(40, 32)
    trajs = [full[f * n:(f + 1) * n] if n <= full.shape[0] // 3 else full[f:f + n] for f in range(3)]
    rng = np.random.default_rng(n)
    kds = [(rng.standard_normal((coils, n)) + 1j * rng.standard_normal((coils, n))).astype(np.complex64) for _ in trajs]
    dcf = rng.uniform(0.2, 1.0, 3 * n).astype(np.float32)
    lut = oracle.kb_lut(4.0, 2.0, 512)
    b = fb.GridBatch(dim, G, 4.0, lut=lut)
    b.set_trajectories(torch.from_numpy(np.concatenate(trajs)).cuda(), [n] * 3)
    kd, dd = torch.from_numpy(np.concatenate([k.ravel() for k in kds])).cuda(), torch.from_numpy(dcf).cuda()
    before = fr.kernel_launches()
    got = b.grid(kd, dd, coils).cpu().numpy()
    # the lanes need the sample-major copy and the scales before the scatter
    assert fr.kernel_launches() - before == (3 if lanes else 1)
    for f, (t, k) in enumerate(zip(trajs, kds)):
        tn = oracle.normalize_traj(np.ascontiguousarray(t), dim, G)[0]
        assert rel_l2(got[f], oracle.grid(tn, dcf[f * n:(f + 1) * n], k, dim, G, 4.0, lut, threads=4)) <= TOL
