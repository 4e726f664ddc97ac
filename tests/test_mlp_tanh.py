"""GPU: the network's tanh alone, point by point against FP64.  All first-layer
units see input 0, the second layer passes one of them on at 2^-14 of its size,
where tanh is the identity to 2^-30, and the output undoes that."""
import numpy as np
import pytest

BOUND = 2  # ulp: what CUDA promises of tanhf


def _net():
    from fastrecon_gb300 import learned_dcf as ld
    p = np.zeros(ld.N_PARAMS, np.float32)
    p[ld.OFF_W1:ld.OFF_B1:ld.N_IN] = 1.0
    p[ld.OFF_W2 + 5 * ld.HIDDEN + 17] = 2.0 ** -14
    p[ld.OFF_W3 + 5] = 2.0 ** 14
    return ld.DCFNet(p)


def _points():
    rng = np.random.default_rng(3)
    split = np.float32(0.65).view(np.uint32) + np.arange(-2000, 2001, dtype=np.int64)
    x = np.concatenate([split.astype(np.uint32).view(np.float32), np.linspace(0, 1, 200001), np.linspace(1, 12, 200001),
                        10.0 ** rng.uniform(-25, 1, 100000), 10.0 ** rng.uniform(1, 38, 1000)]).astype(np.float32)
    return np.concatenate([x, -x])


@pytest.mark.gpu
def test_tanh_points():
    import torch
    x = _points()
    f = np.zeros((x.size, 5), np.float32)
    f[:, 0] = x
    y = _net().forward(torch.from_numpy(f).cuda()).cpu().numpy().astype(np.float64)
    want = np.tanh(x.astype(np.float64))
    ulp = np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
    err = np.abs(y - want) / ulp
    worst = np.argmax(err)
    print("largest error %.3f ulp at %r" % (err[worst], x[worst]))
    assert err[worst] <= BOUND
    assert np.abs(y).max() <= 1


@pytest.mark.gpu
def test_tanh_limits():
    import torch
    tiny = np.float32([0, 1e-45, -1e-45, 1e-40, 1.2e-38, -1e-30])
    x = np.concatenate([tiny, np.float32([np.inf, -np.inf, np.nan, 3.4e38, -3.4e38])])
    f = np.zeros((x.size, 5), np.float32)
    f[:, 0] = x
    y = _net().forward(torch.from_numpy(f).cuda()).cpu().numpy()
    assert np.abs(y[:6] - tiny).max() <= 2.0 ** -100  # below 2^-126 the second layer may flush to zero
    assert np.array_equal(y[6:8], [1, -1]) and np.isnan(y[8]) and np.array_equal(y[9:], [1, -1])
