"""Performance cases: the calls that a program using fastrecon_gb300 makes,
over the range of sizes that they are made with.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare`` makes a program's inputs and the objects it keeps,
``run`` is one pass through the public entry points, ``work`` the bytes and
operations that the pass cannot do without, and ``exact`` the same outputs
from plain torch in 64 bits (taps and table indices as the gridding defines
them in float32: they are part of the definition, not of the rounding).
"""
import math
import os

import numpy as np
import torch

import fastrecon_gb300 as fr
from fastrecon_gb300 import batch as fb
from fastrecon_gb300 import learned_dcf as ld
from fastrecon_gb300 import synth

MODELS = os.path.join(os.path.dirname(os.path.abspath(fr.__file__)), "models")
LUT_LENGTH = 512


def listed():
    return [
        # one frame of a real-time 2D golden-angle series, the smallest call: plan, grid, transform and combine
        # a few thousand samples, where launches and latency are all there is
        dict(name="recon2d_frame", kind="recon", dim=2, family="golden", spokes=21, readout=128, coils=4, recon=64,
             os=2.0, width=4.0),
        # the ordinary 2D radial scan (256 spokes x 512 samples, 8 coils, 512^2 grid)
        dict(name="recon2d_radial", kind="recon", dim=2, family="radial", spokes=256, readout=512, coils=8, recon=256,
             os=2.0, width=4.0),
        # odd everything: a 2D spiral with 5 coils onto an odd 151^2 grid (library transform, shift and combine)
        dict(name="recon2d_spiral_odd", kind="recon", dim=2, family="spiral", spokes=13, readout=1999, coils=5,
             recon=101, os=1.5, width=4.0),
        # a small ragged 3D volume: 3,001 spokes x 101 samples, 3 coils, odd 115^3 grid
        dict(name="recon3d_ragged", kind="recon", dim=3, family="koosh", spokes=3001, readout=101, coils=3, recon=77,
             os=1.5, width=4.0),
        # the largest call: the 3D kooshball, 50,000 spokes x 256 samples, 16 coils, 384^3 grid, 256^3 image
        dict(name="recon3d_kooshball", kind="recon", dim=3, family="koosh", spokes=50000, readout=256, coils=16,
             recon=256, os=1.5, width=4.0),
        # gridding alone with the plan kept: the same trajectory acquired again and again (dynamic 3D, 8 coils)
        dict(name="grid3d_planned", kind="grid", dim=3, family="koosh", spokes=10000, readout=256, coils=8, recon=160,
             os=1.5, width=4.0),
        # batched dynamic spiral: 64 frames of uneven length in one call, 12 coils, 384^2 grids
        dict(name="batch_spiral", kind="batch", dim=2, family="spiral", frames=64, least=4, most=24, readout=2048,
             coils=12, recon=192, os=2.0, width=4.0),
        # the forward model of an iterative recon: a 12-coil image's k-space evaluated on the trajectory
        dict(name="degrid3d", kind="degrid", dim=3, family="koosh", spokes=10000, readout=192, coils=12, recon=128,
             os=1.5, width=4.0),
        # streaming acquisition: 48 new readouts replace old ones and the 16-coil grid follows
        dict(name="update3d", kind="update", dim=3, family="koosh", spokes=4000, readout=256, coils=16, recon=128,
             os=1.5, width=4.0, fresh=48),
        # density compensation by iteration: 20 Pipe-Menon steps for a 3D volume on its 320^3 grid
        dict(name="pipe3d", kind="pipe", dim=3, family="koosh", spokes=12000, readout=256, recon=256, os=1.25,
             width=4.0, iterations=20),
        # density compensation by the trained network: sample counts, features and inference for a 3D volume
        dict(name="learned3d", kind="learned", dim=3, family="koosh", spokes=20000, readout=256, recon=256, os=1.25,
             width=4.0),
        # one step of training that network: loss, gradient and Adam on a mini-batch
        dict(name="train_step", kind="train", batch=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["recon", "recon", "recon", "grid", "batch", "degrid", "update", "pipe", "learned", "train"])
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 1000, 65536))
    width = rng.choice([4.0, 4.0, 4.0, 3.0, 5.0]) if kind in ("recon", "grid", "degrid", "update") else 4.0
    if kind == "batch":
        return dict(kind=kind, dim=2, family="spiral", frames=_log(rng, 4, 64), least=4, most=rng.randint(5, 24),
                    readout=_log(rng, 512, 2048), coils=rng.randint(1, 16), recon=_log(rng, 64, 192),
                    os=rng.choice([1.5, 2.0]), width=width)
    dim = rng.choice([2, 3])
    c = dict(kind=kind, dim=dim, os=rng.choice([1.25, 1.5, 2.0] if dim == 2 else [1.25, 1.5]), width=width)
    if dim == 2:
        c.update(family=rng.choice(["radial", "golden", "spiral"]), readout=_log(rng, 64, 640), recon=_log(rng, 48, 320))
        if c["family"] == "spiral":
            c.update(spokes=_log(rng, 4, 48), readout=_log(rng, 512, 4096))
        else:
            c.update(spokes=_log(rng, 16, 512))
    else:
        c.update(family="koosh", spokes=_log(rng, 400, 20000), readout=_log(rng, 48, 256), recon=_log(rng, 32, 200))
    if kind in ("recon", "grid", "degrid", "update"):
        c["coils"] = rng.randint(1, 32 if dim == 2 else 20)
    if kind == "update":
        c["fresh"] = rng.randint(1, max(1, min(128, c["spokes"] // 4)))
    if kind == "pipe":
        c["iterations"] = rng.randint(3, 20)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rng(seed):
    return np.random.default_rng(seed)


def _lines(directions, readout):
    """Spokes through the centre, k_i = (i - R/2) / R, as (N, 4) float32 on the GPU."""
    k = (torch.arange(readout, device="cuda", dtype=torch.float64) - readout / 2) / readout
    t = torch.zeros((directions.shape[0], readout, 4), device="cuda")
    t[:, :, :directions.shape[1]] = (directions[:, None, :] * k[None, :, None]).float()
    return t.reshape(-1, 4)


def _trajectory(c, rng, spokes=None):
    """The family's trajectory from a seeded start: first angle, or first spoke of the golden sequence."""
    n = spokes or c["spokes"]
    m = torch.arange(n, device="cuda", dtype=torch.float64)
    if c["family"] == "koosh":
        m = m + int(rng.integers(0, 100000))
        cz = (m * synth.GOLDEN_MEANS_3D[0]) % 1.0
        az = 2 * math.pi * ((m * synth.GOLDEN_MEANS_3D[1]) % 1.0)
        sz = torch.sqrt(torch.clamp(1 - cz * cz, min=0))
        return _lines(torch.stack([sz * torch.cos(az), sz * torch.sin(az), cz], 1), c["readout"])
    if c["family"] == "spiral":
        rot = float(rng.uniform(0, 2 * math.pi))
        return torch.from_numpy(synth.spiral_2d(n, c["readout"], rotation=rot)).cuda()
    step = math.pi / n if c["family"] == "radial" else math.pi * (math.sqrt(5) - 1) / 2
    th = m * step + float(rng.uniform(0, math.pi / n))
    return _lines(torch.stack([torch.cos(th), torch.sin(th)], 1), c["readout"])


def _ramp(c, traj):
    """|k| (2D) or |k|^2 (3D), the plain density compensation."""
    q = (traj[:, :c["dim"]].double() ** 2).sum(1)
    return (torch.sqrt(q) if c["dim"] == 2 else q).float()


def _kspace(c, traj, seed):
    """Exact k-space of a seeded phantom seen by smooth coils, with 1 % noise (coils, N)."""
    return synth.kspace(traj.cpu().numpy(), c["dim"], c["recon"], c["coils"], seed=seed % 100003, xp=torch,
                        device="cuda")


def _grid_size(c):
    return int(np.float32(c["recon"]) * np.float32(c["os"]))


def _new_plan(c):
    return fr.GridPlan(c["dim"], _grid_size(c), c["width"], lut_length=LUT_LENGTH, overgrid_factor=c["os"])


def _scan(c, seed):
    traj = _trajectory(c, _rng(seed))
    return traj, _ramp(c, traj), _kspace(c, traj, seed)


def _image_spectrum(c, seed):
    """A coil image's Cartesian k-space (coils, G^d): smooth noise, as an iterative recon holds it."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    G = _grid_size(c)
    r = torch.linspace(-4, 4, G, device="cuda")
    decay = torch.exp(-r.abs())
    shape = (c["coils"],) + (G,) * c["dim"]
    out = torch.complex(torch.randn(shape, generator=g, device="cuda"), torch.randn(shape, generator=g, device="cuda"))
    for d in range(c["dim"]):
        out *= decay.reshape([-1] + [1] * d)
    return out.reshape(c["coils"], -1)


def _batch_frames(c, seed):
    rng = _rng(seed)
    # the scan protocol fixes how many interleaves each frame has
    inter = _rng(3).integers(c["least"], c["most"] + 1, c["frames"])
    trajs = [_trajectory(c, rng, int(k)) for k in inter]
    kd = [_kspace(c, t, seed + f) for f, t in enumerate(trajs)]
    return trajs, [_ramp(c, t) for t in trajs], kd


def _updates(c, traj, seed):
    """Two sets of newly acquired readouts for the block of readouts that streams in."""
    count = c["fresh"] * c["readout"]
    begin = (c["spokes"] // 3) * c["readout"]
    begin = min(begin, traj.shape[0] - count)
    part = traj[begin:begin + count]
    return begin, [_kspace(c, part, seed + 1 + k) for k in range(2)]


def _train_batch(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = c["batch"]
    # features as the volumes give them: log densities at four radii (correlated) and log |k|
    k = torch.rand(n, generator=g, device="cuda") ** (1 / 3)
    base = -2 * torch.log(k + 0.02)
    feats = [base + (0.6 / (i + 1)) * torch.randn(n, generator=g, device="cuda") for i in range(4)]
    feats.append(torch.log(k + 1 / 1024))
    x = torch.stack(feats, 1).contiguous()
    target = -base + 0.1 * torch.randn(n, generator=g, device="cuda")
    weight = torch.rand(n, generator=g, device="cuda") * 2
    m = 1e-2 * torch.randn(ld.N_PARAMS, generator=g, device="cuda")
    v = 1e-4 * (0.1 + torch.rand(ld.N_PARAMS, generator=g, device="cuda"))
    return x, target, weight, m, v


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "train":
        x, target, weight, m, v = _train_batch(c, seed)
        net = ld.DCFNet(seed=seed % 1000)
        net.m.copy_(m)  # in the middle of a training run
        net.v.copy_(v)
        net.step = 200
        return dict(kind=kind, net=net, x=x, target=target, weight=weight)
    if kind == "batch":
        trajs, dcfs, kd = _batch_frames(c, seed)
        counts = [t.shape[0] for t in trajs]
        traj = torch.cat(trajs)
        b = fb.GridBatch(c["dim"], _grid_size(c), c["width"], lut_length=LUT_LENGTH, overgrid_factor=c["os"])
        b.set_trajectories(traj, counts)
        out = torch.empty((c["frames"], c["coils"], _grid_size(c) ** c["dim"]), dtype=torch.complex64, device="cuda")
        return dict(kind=kind, batch=b, kd=torch.cat([k.reshape(-1) for k in kd]), dcf=torch.cat(dcfs),
                    coils=c["coils"], out=out)
    if kind == "recon":
        traj, dcf, kd = _scan(c, seed)
        rec = fr.Recon(c["dim"], c["recon"], c["os"], c["coils"], kernel_width=c["width"], lut_length=LUT_LENGTH,
                       max_samples=traj.shape[0])
        img = torch.empty(c["recon"] ** c["dim"], dtype=torch.float32, device="cuda")
        return dict(kind=kind, recon=rec, traj=traj, dcf=dcf, kd=kd, out=img)
    plan = _new_plan(c)
    if kind in ("pipe", "learned"):
        traj = _trajectory(c, _rng(seed))
        plan.set_trajectory(traj)
        s = dict(kind=kind, plan=plan, traj=traj)
        if kind == "pipe":
            s["iterations"] = c["iterations"]
        else:
            s["net"] = ld.DCFNet.load(os.path.join(MODELS, "dcf_mlp_%dd.npz" % c["dim"]))
        return s
    if kind == "degrid":
        traj = _trajectory(c, _rng(seed))
        plan.set_trajectory(traj)
        out = torch.empty((c["coils"], traj.shape[0]), dtype=torch.complex64, device="cuda")
        return dict(kind=kind, plan=plan, grid=_image_spectrum(c, seed), out=out)
    traj, dcf, kd = _scan(c, seed)
    plan.set_trajectory(traj)
    grid = torch.empty((c["coils"], plan.cells), dtype=torch.complex64, device="cuda")
    if kind == "grid":
        return dict(kind=kind, plan=plan, kd=kd, dcf=dcf, out=grid)
    begin, news = _updates(c, traj, seed)
    plan.grid(kd, dcf, out=grid)
    return dict(kind=kind, plan=plan, kd=kd, dcf=dcf, grid=grid, begin=begin, news=news, turn=0)


def run(state):
    s = state
    kind = s["kind"]
    if kind == "recon":
        return s["recon"].run(s["traj"], s["dcf"], s["kd"], out=s["out"])
    if kind == "grid":
        return s["plan"].grid(s["kd"], s["dcf"], out=s["out"])
    if kind == "batch":
        return s["batch"].grid(s["kd"], s["dcf"], s["coils"], out=s["out"])
    if kind == "degrid":
        return s["plan"].degrid(s["grid"], out=s["out"])
    if kind == "update":
        new = s["news"][s["turn"]]
        s["turn"] ^= 1
        s["plan"].update(s["kd"], new, s["begin"], s["dcf"], s["grid"])
        return s["grid"], s["kd"]
    if kind == "pipe":
        return s["plan"].dcf_pipe(s["iterations"])
    if kind == "learned":
        return ld.learned_dcf(s["plan"], s["traj"], s["net"])
    net = s["net"]
    loss = net.loss_grad(s["x"], s["target"], s["weight"])
    net.adam(lr=1e-3)
    return dict(loss=loss, grad=net.grad, master=net.master, bf16=net.bf16, m=net.m, v=net.v)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _taps(c):
    """Mean taps of a sample: the kernel ball's volume."""
    hw = c["width"] / 2
    return math.pi * hw * hw if c["dim"] == 2 else 4 / 3 * math.pi * hw ** 3


def work(case):
    c = case
    kind = c["kind"]
    h, i = ld.HIDDEN, ld.N_IN
    net_flops = 2 * (i * h + h * h + h)
    if kind == "train":
        # master, m and v read and written, gradient and 16-bit copy written; forward and two backward products
        return {"bytes": 4 * c["batch"] * (i + 2) + ld.N_PARAMS * (6 * 4 + 4 + 2), "flops": 3 * net_flops * c["batch"]}
    G = _grid_size(c)
    cells = G ** c["dim"]
    if kind == "batch":
        n = c["frames"] * (c["least"] + c["most"]) // 2 * c["readout"]
        return {"bytes": n * (16 + 4 + 8 * c["coils"]) + c["frames"] * c["coils"] * cells * 8,
                "flops": 4 * _taps(c) * n * c["coils"]}
    n = c["spokes"] * c["readout"]
    if kind == "recon":
        fft = 5 * c["coils"] * cells * math.log2(cells)
        return {"bytes": n * (16 + 4 + 8 * c["coils"]) + 4 * c["recon"] ** c["dim"],
                "flops": 4 * _taps(c) * n * c["coils"] + fft}
    if kind in ("grid", "degrid"):
        extra = 4 if kind == "grid" else 0
        return {"bytes": n * (16 + extra + 8 * c["coils"]) + c["coils"] * cells * 8,
                "flops": 4 * _taps(c) * n * c["coils"]}
    if kind == "update":
        m = c["fresh"] * c["readout"]
        touched = min(cells, m * 2 ** c["dim"])  # a readout advances about one cell a sample
        return {"bytes": m * (16 + 4 + 3 * 8 * c["coils"]) + touched * c["coils"] * 16,
                "flops": 4 * _taps(c) * m * c["coils"]}
    if kind == "pipe":
        return {"bytes": c["iterations"] * (n * (2 * 16 + 3 * 4) + 2 * cells * 4),
                "flops": c["iterations"] * 4 * _taps(c) * n}
    return {"bytes": n * (2 * 16 + 4) + cells * 4, "flops": n * net_flops}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _lut(c):
    """The Kaiser-Bessel table: rounding steps as the method defines them (Beatty's beta, float32 radii)."""
    f = np.float32
    w, a = f(c["width"]), f(c["os"])
    wa = f(w * w) / f(a * a)
    beta = float(f(math.pi * math.sqrt(float(wa) * (float(a) - 0.5) * (float(a) - 0.5) - 0.8)))
    dk = f(float(w) / 2.0 / (LUT_LENGTH - 1))
    k = (dk * np.arange(LUT_LENGTH, dtype=f)).astype(f)
    r = (f(2) * k / w).astype(f).astype(np.float64)
    i0 = torch.special.i0(torch.from_numpy(beta * np.sqrt(1 - r * r))).numpy()
    out = (i0 / float(w)).astype(f)
    return torch.from_numpy((out / out[0]).astype(f)).cuda()


def _normalized(c, traj):
    lo, hi = traj[:, 0].min(), traj[:, 0].max()
    scale = torch.tensor(float(_grid_size(c) - 1), device="cuda") / (hi - lo)
    return (traj[:, :c["dim"]] + (-lo)) * scale


def _for_taps(c, pos, lut, visit):
    """visit(rows, cells, weights) for every tap: cells row-major with x fastest, float32 geometry, 64-bit weights."""
    d, G = c["dim"], _grid_size(c)
    hw = torch.tensor(c["width"] / 2, device="cuda", dtype=torch.float32)
    start = torch.ceil(pos - hw).to(torch.int64).clamp(min=0)
    end = torch.floor(pos + hw).to(torch.int64).clamp(max=G - 1)
    F = int(math.floor(c["width"])) + 1
    w64 = lut.double()
    for o in range(F ** d):
        off = [(o // F ** a) % F for a in range(d)]
        cell = [start[:, a] + off[a] for a in range(d)]
        diff = [cell[a].float() - pos[:, a] for a in range(d)]
        s2 = diff[1] * diff[1]
        if d == 3:
            s2 = diff[2] * diff[2] + s2
        dk = torch.sqrt(s2 + diff[0] * diff[0])
        ok = dk < hw
        for a in range(d):
            ok &= cell[a] <= end[:, a]
        rows = torch.nonzero(ok).squeeze(1)
        if rows.numel() == 0:
            continue
        q = (dk[rows] / hw) * float(LUT_LENGTH - 1)
        index = torch.floor(q.double() + 0.5).to(torch.int64)
        flat = cell[d - 1][rows]
        for a in range(d - 2, -1, -1):
            flat = flat * G + cell[a][rows]
        visit(rows, flat, w64[index])


def _chunks(n, size=1 << 19):
    return [(b, min(b + size, n)) for b in range(0, n, size)]


def _grid64(c, pos, values):
    """values: (N, K) float64 -> (cells, K) float64."""
    lut = _lut(c)
    grid = torch.zeros((_grid_size(c) ** c["dim"], values.shape[1]), dtype=torch.float64, device="cuda")
    for b, e in _chunks(pos.shape[0]):
        v = values(b, e) if callable(values) else values[b:e]
        _for_taps(c, pos[b:e], lut, lambda rows, cells, w: grid.index_add_(0, cells, v[rows] * w[:, None]))
    return grid


class _Samples:
    """dcf x k-space rows (sample, re / im of every coil) in 64 bits, made a block at a time."""

    def __init__(self, dcf, kd):
        self.dcf, self.kd, self.shape = dcf, kd, (kd.shape[1], 2 * kd.shape[0])

    def __call__(self, b, e):
        v = torch.view_as_real(self.kd[:, b:e].t().contiguous()).double()
        return (v * self.dcf[b:e].double()[:, None, None]).reshape(e - b, -1)


def _gridded64(c, traj, dcf, kd):
    g = _grid64(c, _normalized(c, traj), _Samples(dcf, kd))
    return torch.view_as_complex(g.reshape(g.shape[0], -1, 2))  # (cells, coils)


def _degrid64(c, pos, grid):
    """grid: (cells, K) float64 -> (N, K) float64."""
    lut = _lut(c)
    out = torch.zeros((pos.shape[0], grid.shape[1]), dtype=torch.float64, device="cuda")
    for b, e in _chunks(pos.shape[0]):
        part = out[b:e]
        _for_taps(c, pos[b:e], lut, lambda rows, cells, w: part.index_add_(0, rows, grid[cells] * w[:, None]))
    return out


def _shift(img):
    """The shift of the image by half its size; for odd sizes the swaps in their order (they overlap)."""
    sizes = img.shape
    if all(n % 2 == 0 for n in sizes):
        return torch.fft.fftshift(img)
    sy, sx = sizes[-2:]
    hy, hx = sy // 2, sx // 2
    to_y = [y + hy if y < hy else y - hy for y in range(sy)]
    to_x = [x + hx if x < hx else x - hx for x in range(sx)]
    if len(sizes) == 2:
        at = list(range(sy * sx))
        for y in range(hy):
            for x in range(sx):
                i, j = y * sx + x, (y + hy) * sx + to_x[x]
                at[i], at[j] = at[j], at[i]
        return img.reshape(-1)[torch.tensor(at, device=img.device)].reshape(sizes)
    plane = sy * sx
    at = list(range(2 * plane))  # a plane and the one half the size above it
    for y in range(sy):
        for x in range(sx):
            i, j = y * sx + x, plane + to_y[y] * sx + to_x[x]
            at[i], at[j] = at[j], at[i]
    at = torch.tensor(at, device=img.device)
    out = img.clone()
    h = sizes[0] // 2
    both = torch.stack([img[:h], img[h:2 * h]], 1).reshape(h, 2 * plane)[:, at].reshape(h, 2, sy, sx)
    out[:h], out[h:2 * h] = both[:, 0], both[:, 1]
    return out


def _recon64(c, traj, dcf, kd):
    G, R = _grid_size(c), c["recon"]
    g = _gridded64(c, traj, dcf, kd)
    o = (G - R) // 2
    total = torch.zeros((R,) * c["dim"], dtype=torch.float64, device="cuda")
    for k in range(g.shape[1]):
        img = torch.fft.ifftn(g[:, k].reshape((G,) * c["dim"]).contiguous(), norm="forward")
        img = _shift(img)[(slice(o, o + R),) * c["dim"]]
        total += img.real ** 2 + img.imag ** 2
    return torch.sqrt(total).reshape(-1)


def _network64(params, x):
    p = params.double()
    w1 = p[ld.OFF_W1:ld.OFF_B1].reshape(ld.HIDDEN, ld.N_IN)
    w2 = p[ld.OFF_W2:ld.OFF_B2].reshape(ld.HIDDEN, ld.HIDDEN)
    h1 = torch.tanh(x @ w1.t() + p[ld.OFF_B1:ld.OFF_W2])
    h2 = torch.tanh(h1 @ w2.t() + p[ld.OFF_B2:ld.OFF_W3])
    return h2 @ p[ld.OFF_W3:ld.OFF_B3] + p[ld.OFF_B3]


def _learned64(c, traj):
    G, d = _grid_size(c), c["dim"]
    cell = torch.floor(_normalized(c, traj) + 0.5).to(torch.int64).clamp(0, G - 1)
    flat = cell[:, d - 1]
    for a in range(d - 2, -1, -1):
        flat = flat * G + cell[:, a]
    table = torch.bincount(flat, minlength=G ** d).reshape((G,) * d)
    for a in range(d):
        table = torch.cumsum(table, a)
    table = torch.nn.functional.pad(table, (1, 0) * d)  # prefix sums with a row of zeros in front
    feats = []
    for r in ld.RADII:
        count = torch.zeros(traj.shape[0], dtype=torch.int64, device="cuda")
        for corner in range(2 ** d):
            at, sign = [], 1
            for a in range(d):
                if (corner >> a) & 1:
                    at.append((cell[:, a] - r).clamp(min=0))
                    sign = -sign
                else:
                    at.append((cell[:, a] + r).clamp(max=G - 1) + 1)
            count += sign * table[tuple(at[::-1])]
        feats.append(torch.log(count.double() / (2 * r + 1) ** d))
    k = torch.sqrt((traj[:, :d].double() ** 2).sum(1))
    feats.append(torch.log(k / k.max() + 1 / 1024))
    x = torch.stack(feats, 1)
    z = np.load(os.path.join(MODELS, "dcf_mlp_%dd.npz" % d))
    y = _network64(torch.from_numpy(np.asarray(z["params"], np.float32)).cuda().bfloat16(), x)
    if "residual" in z.files and int(z["residual"]):
        y = y - x[:, 1]
    # divided by the square of the kernel's mass over the plane or space
    steps = 100000
    hw = c["width"] / 2
    r = (np.arange(steps) + 0.5) * (hw / steps)
    w = _lut(c).double().cpu().numpy()
    at = w[np.minimum(np.rint(r / hw * (LUT_LENGTH - 1)).astype(np.int64), LUT_LENGTH - 1)]
    mass = float(np.sum(at * (2 * np.pi * r if d == 2 else 4 * np.pi * r * r)) * (hw / steps))
    return torch.exp(y) / mass ** 2


def _train64(c, seed):
    x, target, weight, m, v = (t.double() for t in _train_batch(c, seed))
    master = torch.from_numpy(ld.DCFNet.init_params(seed % 1000)).cuda()
    p = master.bfloat16().double().requires_grad_()
    r = _network64(p, x) - target
    loss = (weight * r * r).mean()
    loss.backward()
    g, step = p.grad, 201
    m = 0.9 * m + 0.1 * g
    v = 0.999 * v + 0.001 * g * g
    new = master.double() - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return dict(loss=loss.detach().reshape(1), grad=g, master=new, bf16=None, m=m, v=v)


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "train":
        return _train64(c, seed)
    if kind == "batch":
        trajs, dcfs, kd = _batch_frames(c, seed)
        return torch.stack([_gridded64(c, *f).t().contiguous() for f in zip(trajs, dcfs, kd)])
    traj = _trajectory(c, _rng(seed))
    if kind == "learned":
        return _learned64(c, traj)
    if kind == "degrid":
        pos, grid = _normalized(c, traj), _image_spectrum(c, seed)
        out = _degrid64(c, pos, torch.view_as_real(grid.t().contiguous()).double().reshape(grid.shape[1], -1))
        return torch.view_as_complex(out.reshape(pos.shape[0], -1, 2)).t().contiguous()
    if kind == "pipe":
        pos = _normalized(c, traj)
        w = torch.ones((traj.shape[0], 1), dtype=torch.float64, device="cuda")
        for _ in range(c["iterations"]):
            p = _degrid64(c, pos, _grid64(c, pos, w))
            w = torch.where(p > 0, w / p, w)
        return w.squeeze(1)
    dcf, kd = _ramp(c, traj), _kspace(c, traj, seed)
    if kind == "recon":
        return _recon64(c, traj, dcf, kd)
    if kind == "update":
        begin, news = _updates(c, traj, seed)
        kd[:, begin:begin + news[0].shape[1]] = news[0]
        return _gridded64(c, traj, dcf, kd).t().contiguous(), None
    return _gridded64(c, traj, dcf, kd).t().contiguous()
