"""The Gaussian where the number of planes a warp walks changes (3, 6, 15), with depths that end
within a turn of three planes -- against the oracle, bit for bit."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

# 1 to 8 column blocks a plane: at most and more than 444 blocks with 3 planes, and 592 with 6
SHAPES = [(1332, 16, 32), (1333, 16, 32), (3552, 15, 30), (3553, 16, 20), (166, 33, 63), (167, 60, 60), (444, 60, 50),
          (445, 60, 50)]


@pytest.mark.parametrize("shape", SHAPES)
def test_gaussian_walk(orc, shape):
    rng = np.random.default_rng(3)
    v = rng.normal(0, 100, shape).astype(np.float32)
    assert np.array_equal(tb.gaussian(v, 1).view(np.uint32), orc.gaussian(v, 1).view(np.uint32))
    u = (rng.random(shape) * 3000).astype(np.uint16)
    u[rng.random(shape) < 0.5] = 0
    assert np.array_equal(tb.subject_image_pre(u), orc.subject_image_pre(u.astype(np.float32)))
