"""The CDM passes on volumes of few voxels on some axis, whose rows and planes fill little of the
blocks and tiles of ordinary ones, on both sides of each line between two forms of a pass --
against the oracle, bit for bit."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

# more planes than clusters take; planes of 1 to 1600 voxels; rows of one and two voxels with and
# without padding; one plane; planes that use 77, 78, 80 and 95 % of the threads that walk them
POISSON = [(300, 1, 1), (70, 1, 2), (66, 3, 2), (65, 40, 1), (70, 2, 3), (90, 4, 4), (67, 5, 6), (66, 7, 30), (70, 1, 37),
           (1, 1, 5000), (1, 1100, 1), (1, 1030, 2), (1, 1100, 5), (3, 1030, 2), (66, 28, 28), (66, 40, 40), (66, 41, 20),
           (66, 44, 44), (70, 16, 16), (200, 8, 64), (3000, 1, 2), (900, 7, 1), (1500, 3, 2), (70, 600, 2)]


@pytest.mark.parametrize("shape", POISSON)
def test_poisson_thin(orc, shape):
    rng = np.random.default_rng(sum(shape))
    d = rng.normal(0, 1, shape + (3,)).astype(np.float32)
    d[rng.random(shape) < 0.3] = 0
    d[rng.random(shape) < 0.1] = -0.0
    assert np.array_equal(tb.cdm_poisson(d).view(np.uint32), orc.cdm_poisson(d).view(np.uint32))


# one level each (no axis is longer than min_dimension); rows of two voxels are not padded
LEVELS = [(70, 8, 8), (70, 33, 2), (66, 7, 2), (70, 3, 5), (300, 2, 4), (150, 2, 2), (2, 1100, 2), (65, 2, 300),
          (70, 16, 16), (66, 13, 90), (70, 12, 20)]


def thin_pair(shape, seed):
    """A smooth random texture, and the same moved by a voxel and a half along the longest axis."""
    rng = np.random.default_rng(seed)
    v = rng.normal(0, 1, shape)
    for ax, n in enumerate(shape):
        for _ in range(3 if n >= 8 else 0):
            v = v + np.roll(v, 1, ax) + np.roll(v, -1, ax)
    v = (v - v.min()) / (v.max() - v.min()) * 200 + 20
    ax = int(np.argmax(shape))
    m = 0.5 * (np.roll(v, 1, ax) + np.roll(v, 2, ax)) + rng.normal(0, 1, shape)
    return v, np.clip(m, 0, 255)


@pytest.mark.parametrize("gtype", ["r", "d"])
@pytest.mark.parametrize("u8", [True, False])
@pytest.mark.parametrize("shape", LEVELS)
def test_levels_of_thin_volumes(orc, shape, u8, gtype):
    """Whole levels: the field and the number of iterations.  Where an axis has only a few voxels
    no field is better than none and the result is zero, but the costs of the fields on the way
    decide how many iterations there are."""
    It, Is = (v.astype(np.uint8 if u8 else np.float32) for v in thin_pair(shape, sum(shape)))
    kw = dict(resolution=1.0, min_dimension=64, gradient_type=gtype)
    od, ook, iters = orc.cdm(It, Is, **kw)
    d = np.ones(shape + (3,), np.float32)
    with tb.Engine() as eng:
        r = eng.wait(eng.submit(Is, fixed=It, linear=False, cdm=True, cdm_param=tb.reg.cdm_param(**kw), field_out=d))
    assert r["status"] == 0 and bool(r["cdm_ok"]) == ook
    assert r["cdm_iterations"] == iters
    assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
    p, ok = tb.reg.cdm(It, Is, tb.reg.cdm_param(**kw))
    assert ok == ook and np.array_equal(p.view(np.uint32), od.view(np.uint32))


# on both sides of the lines between tiles and a voxel a thread, and between tiles of 2 and of 8
# planes: few voxels on one axis and on two, below and above 200000 voxels
GRADIENT = [(1, 1, 300), (1, 300, 1), (300, 1, 1), (30, 40, 1), (40, 30, 2), (60, 60, 3), (60, 60, 8), (60, 60, 12),
            (1, 64, 80), (2, 70, 70), (3, 60, 60), (40, 1, 50), (40, 2, 50), (60, 3, 60), (60, 5, 60), (100, 8, 8),
            (700, 300, 1), (300, 230, 3), (180, 170, 7), (160, 160, 8), (150, 150, 9), (1, 450, 450), (2, 320, 320),
            (3, 260, 260), (300, 1, 700), (300, 2, 340), (300, 2, 300), (300, 3, 230), (3200, 8, 8), (1500, 12, 12)]


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("shape", GRADIENT)
def test_gradient_thin(orc, shape, dtype):
    """The mean cost to a float ulp: its double sum runs in another order."""
    rng = np.random.default_rng(sum(shape))
    J, I = ((rng.random(shape) * 255).astype(dtype) for _ in range(2))
    J[rng.random(shape) < 0.2] = 0
    I[rng.random(shape) < 0.2] = 0
    field, cost = tb.cdm_gradient(J, I)
    ofield, ocost = orc.cdm_gradient(J, I)[:2]
    assert np.array_equal(field.view(np.uint32), np.asarray(ofield, np.float32).view(np.uint32))
    assert abs(cost - ocost) <= np.spacing(np.float32(abs(ocost)))


@pytest.mark.parametrize("shape", [(40, 30, 2), (1, 64, 80), (300, 230, 3)])
def test_gradient_thin_float_extremes(orc, shape):
    """Denormal, huge and infinite pixels: the same field, NaN where the oracle has NaN."""
    rng = np.random.default_rng(7)
    J, I = ((rng.random(shape) * 255).astype(np.float32) for _ in range(2))
    for v in (1e-42, 1e30, np.inf, -np.inf, -3.0):
        J[rng.random(shape) < 0.002] = v
        I[rng.random(shape) < 0.002] = v
    field, _ = tb.cdm_gradient(J, I)
    ofield = np.asarray(orc.cdm_gradient(J, I)[0], np.float32)
    nan = np.isnan(ofield)
    assert np.array_equal(np.isnan(field), nan)
    assert np.array_equal(field[~nan].view(np.uint32), ofield[~nan].view(np.uint32))
