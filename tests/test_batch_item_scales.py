"""GPU: a coil that is strong in one part of k-space and weak in another keeps
its precision in both, whatever the other coils do there: a batch's fixed-point
scales are per work item and coil."""
import numpy as np
import pytest

from conftest import rel_l2
from fastrecon_gb300 import synth

TOL = 1e-5  # FP32 values, sums exact to 2^-22 of the coil's largest value in the item


@pytest.mark.gpu
@pytest.mark.parametrize("tile,coil_group,coils", [((0, 0, 0), 0, 12), ((16, 16, 0), 8, 8), ((32, 32, 0), 16, 17),
                                                   ((16, 16, 0), 4, 3)])
@pytest.mark.parametrize("weak", [1e-3, 1e-6, 1e-9])
def test_unevenly_weak_coil(oracle, tile, coil_group, coils, weak):
    import torch

    from fastrecon_gb300 import batch as fb
    G, width = 128, 4.0
    trajs = [synth.radial_2d(201, 128), synth.golden_angle_2d(90, 100)]
    rng = np.random.default_rng(coils)
    lut = oracle.kb_lut(width, 2.0, 512)
    norm = [oracle.normalize_traj(t, 2, G)[0] for t in trajs]
    dcfs = [rng.uniform(0.2, 1.0, t.shape[0]).astype(np.float32) for t in trajs]
    kds = [(rng.standard_normal((coils, t.shape[0])) + 1j * rng.standard_normal((coils, t.shape[0]))).astype(np.complex64)
           for t in trajs]
    for k, tn in zip(kds, norm):
        k[1, tn[:, 1] < G // 2] *= np.float32(weak)
        k[2, tn[:, 1] >= G // 2] *= np.float32(weak)
    b = fb.GridBatch(2, G, width, lut=lut, tile=tile, coil_group=coil_group)
    b.set_trajectories(torch.from_numpy(np.concatenate(trajs)).cuda(), [t.shape[0] for t in trajs])
    got = b.grid(torch.from_numpy(np.concatenate([k.ravel() for k in kds])).cuda(),
                 torch.from_numpy(np.concatenate(dcfs)).cuda(), coils).cpu().numpy()
    # rows of cells whose tiles (edges of at most 32 cells) hold only samples of one half
    low, high = slice(0, G // 2 - 34), slice(G // 2 + 34, G)
    for f in range(2):
        want = oracle.grid_f64(norm[f], dcfs[f], kds[f], 2, G, width, lut).reshape(coils, G, G)
        have = got[f].reshape(coils, G, G)
        for c in range(coils):
            for rows in (low, high):
                assert rel_l2(have[c][rows], want[c][rows]) <= TOL, (f, c, rows)
