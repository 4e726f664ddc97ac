"""GPU: the plan's bins, work items and bounds over tile and record counts on both
sides of the one-launch count scan (at most 4096 tiles and 2^22 possible
records; a block per 256 tiles), whole numbers and bits equal to the oracle."""
import numpy as np
import pytest

from conftest import rel_l2


def _trajectory(dim, n, rng):
    t = np.zeros((n, 4), np.float32)
    t[:, :dim] = rng.uniform(-0.5, 0.5, (n, dim)) * rng.uniform(0, 1, (n, 1)) ** 3  # dense centre: split tiles
    if n > 1:
        t[0, :dim], t[1, :dim] = -0.5, 0.5
    return t


def _want_bins(oracle, norm, dim, G, W, tile, nt):
    s, e = oracle.sample_range(norm, dim, G, W / 2)
    lo, hi = oracle.sample_tiles(s, e, dim, tile)
    keep = np.nonzero(lo[:, 0] <= hi[:, 0])[0]
    tiles, smp = [], []
    span = (hi[keep] - lo[keep]).max(axis=0) if len(keep) else (0, 0, 0)
    for dz in range(span[2] + 1):
        for dy in range(span[1] + 1):
            for dx in range(span[0] + 1):
                p = lo[keep] + (dx, dy, dz)
                ok = (p <= hi[keep]).all(axis=1)
                tiles.append(((p[ok, 2] * nt[1] + p[ok, 1]) * nt[0] + p[ok, 0]).astype(np.int64))
                smp.append(keep[ok])
    tiles, smp = np.concatenate(tiles), np.concatenate(smp)
    o = np.lexsort((smp, tiles))
    return tiles[o], smp[o]


@pytest.mark.gpu
@pytest.mark.parametrize("dim,G,tile", [(2, 31, 32), (2, 60, 4), (2, 64, 4), (2, 66, 4), (2, 255, 4), (2, 260, 4),
                                        (3, 50, 8), (3, 128, 8), (3, 129, 8)])
@pytest.mark.parametrize("n", [0, 1, 31, 1025, 5000])
def test_counts(oracle, dim, G, tile, n):
    import fastrecon_gb300 as fr
    import torch
    W, chunk = 4.0, 64
    tile = (tile, tile, tile if dim == 3 else 1)
    nt = [-(-G // tile[0]), -(-G // tile[1]), -(-G // tile[2]) if dim == 3 else 1]
    rng = np.random.default_rng(n + G)
    p = fr.GridPlan(dim, G, W, tile=tile, coil_group=16, chunk=chunk)
    for _ in range(2):  # a second trajectory reuses the counters
        traj = _trajectory(dim, n, rng)
        p.set_trajectory(torch.from_numpy(traj).cuda())
    norm, tr, sc, nlo, nhi = oracle.normalize_traj(traj, dim, G)
    rlo, rhi = oracle.comp_bounds(traj, dim)
    got = p.bounds()
    for a, b in zip(got, (rlo, rhi, nlo, nhi)):
        a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
        same = a.view(np.uint32) == b.view(np.uint32)
        assert np.all(same | (np.isnan(a) & np.isnan(b)))  # a NaN's payload is the machine's own
    off, pairs = (x.cpu().numpy() for x in p.bins())
    stats = p.stats()
    if n < 2:  # one sample: the scale is infinite, its cell not a number
        counts = np.diff(off)
        assert n == 0 and len(pairs) == 0 or n == 1
    else:
        wt, ws = _want_bins(oracle, norm, dim, G, W, tile, nt)
        counts = np.bincount(wt, minlength=nt[0] * nt[1] * nt[2])
        assert np.array_equal(off, np.concatenate([[0], np.cumsum(counts)]))
        gt = np.repeat(np.arange(len(counts)), counts)
        o = np.lexsort((pairs, gt))
        assert np.array_equal(pairs[o], ws)
    items = -(-counts // chunk)
    assert stats["tiles"] == len(counts) and stats["pairs"] == counts.sum()
    assert stats["items"] == np.maximum(items, 1).sum() and stats["slots"] == items[items > 1].sum()
    if n >= 2 and G <= 66:
        kd = (rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n))).astype(np.complex64)
        dcf = rng.uniform(0.5, 1.5, n).astype(np.float32)
        g = p.grid(torch.from_numpy(kd).cuda(), torch.from_numpy(dcf).cuda()).cpu().numpy()
        assert rel_l2(g, oracle.grid(norm, dcf, kd, dim, G, W, p.lut, threads=4)) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(1 << 20) - 7, (1 << 20) + 7])
def test_many_records(oracle, n):
    """2^22 possible records: four tiles a sample in 2D."""
    import fastrecon_gb300 as fr
    import torch
    traj = _trajectory(2, n, np.random.default_rng(5))
    p = fr.GridPlan(2, 200, 4.0)
    p.set_trajectory(torch.from_numpy(traj).cuda())
    norm = oracle.normalize_traj(traj, 2, 200)[0]
    off, pairs = (x.cpu().numpy() for x in p.bins())
    wt, ws = _want_bins(oracle, norm, 2, 200, 4.0, (32, 32, 1), [7, 7, 1])
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(wt, minlength=49))]))
    gt = np.repeat(np.arange(49), np.diff(off))
    assert np.array_equal(pairs[np.lexsort((pairs, gt))], ws)
