"""GPU tests of what an affine cost prepares on the device (REGB_COST_MI, REGB_COST_CORR).

Widths around the eight voxels a thread of the moving volume's half texture converts,
volumes around the sixteen voxels a load of the fixed volume's statistics takes, and
volumes that start at an odd address.  Joint counts and the correlation cost (exact
moments) are compared bit for bit; the MI cost is a double sum of 65536 terms added in
another order, within 1e-12 relative (the bar of the other cost tests).
"""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu


def _volumes(shape, seed):
    rng = np.random.default_rng(seed)
    v = rng.integers(0, 256, (2,) + shape).astype(np.uint8)
    v[rng.random(v.shape) < 0.4] = 0
    Ts = np.array([np.r_[(np.eye(3) + rng.normal(0, 0.02, (3, 3))).ravel(), rng.normal(0, 0.4, 3)] for _ in range(3)],
                  np.float32)
    Ts[0] = np.r_[np.eye(3).ravel(), 0, 0, 0]
    return v[0], v[1], Ts


def _check(orc, f, m, Ts, fd, md):
    cost, hist = tb.mi_cost(fd, md, Ts, return_hist=True)
    corr = tb.corr_cost(fd, md, Ts)
    for k, T in enumerate(Ts):
        assert np.array_equal(hist[k], orc.mi_hist(f, m, T))
        assert cost[k] == pytest.approx(orc.mi_cost(f, m, T), rel=1e-12, abs=1e-12)
        assert corr[k] == orc.corr_cost(f, m, T)


@pytest.mark.parametrize("shape", [(2, 2, 3), (3, 5, 7), (2, 3, 8), (5, 4, 9), (11, 13, 17), (33, 37, 40)])
def test_set_up_of_odd_sizes(orc, shape):
    f, m, Ts = _volumes(shape, 3)
    _check(orc, f, m, Ts, f, m)


@pytest.mark.parametrize("off", [1, 7, 16])
def test_set_up_of_volumes_at_any_address(orc, off):
    import torch

    f, m, Ts = _volumes((12, 19, 23), 4)
    buf = torch.zeros(2, off + f.size, dtype=torch.uint8, device="cuda")
    dev = []
    for b, v in zip(buf, (f, m)):
        b[off:].copy_(torch.from_numpy(v).reshape(-1))
        dev.append(b[off:].view(v.shape))
    _check(orc, f, m, Ts, *dev)
