"""The tiled 'r' gradients (cdm_gradient, reg/cdm.hpp:46-78) at the edges of their tiles and
on either side of the size where the tile changes, against the oracle: the field bit for
bit, the mean cost to a float ulp (its double sum runs in another order)."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 7, 31), (3, 8, 32), (4, 9, 33), (5, 1, 65), (1, 17, 40), (8, 8, 64), (9, 16, 36),
          (17, 40, 95), (50, 63, 63), (47, 64, 67), (40, 72, 70)]


def volumes(shape, dtype, rng):
    J, I = ((rng.random(shape) * 255).astype(dtype) for _ in range(2))
    J[rng.random(shape) < 0.2] = 0
    I[rng.random(shape) < 0.2] = 0
    return J, I


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_gradient_tiles(orc, shape, dtype):
    J, I = volumes(shape, dtype, np.random.default_rng(sum(shape)))
    for gtype in "rd":
        field, cost = tb.cdm_gradient(J, I, gtype)
        ofield, ocost = orc.cdm_gradient(J, I, gtype)[:2]
        assert np.array_equal(field.view(np.uint32), np.asarray(ofield, np.float32).view(np.uint32))
        assert abs(cost - ocost) <= np.spacing(np.float32(abs(ocost)))


@pytest.mark.parametrize("shape", [(9, 16, 36), (40, 72, 70)])
def test_gradient_float_extremes(orc, shape):
    """Denormal, huge and infinite pixels: the same field, NaN where the oracle has NaN."""
    rng = np.random.default_rng(7)
    J, I = volumes(shape, np.float32, rng)
    for v in (1e-42, 1e30, np.inf, -np.inf, -3.0):
        J[rng.random(shape) < 0.002] = v
        I[rng.random(shape) < 0.002] = v
    field, _ = tb.cdm_gradient(J, I)
    ofield = np.asarray(orc.cdm_gradient(J, I)[0], np.float32)
    nan = np.isnan(ofield)
    assert np.array_equal(np.isnan(field), nan)
    assert np.array_equal(field[~nan].view(np.uint32), ofield[~nan].view(np.uint32))
