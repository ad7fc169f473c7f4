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
           (66, 44, 44), (70, 16, 16), (200, 8, 64)]


@pytest.mark.parametrize("shape", POISSON)
def test_poisson_thin(orc, shape):
    rng = np.random.default_rng(sum(shape))
    d = rng.normal(0, 1, shape + (3,)).astype(np.float32)
    d[rng.random(shape) < 0.3] = 0
    d[rng.random(shape) < 0.1] = -0.0
    assert np.array_equal(tb.cdm_poisson(d).view(np.uint32), orc.cdm_poisson(d).view(np.uint32))


# one level each (no axis is longer than min_dimension); rows of two voxels are not padded
LEVELS = [(70, 8, 8), (70, 33, 2), (66, 7, 2), (70, 3, 5), (300, 2, 4), (150, 2, 2), (2, 1100, 2), (65, 2, 300), (3, 2, 700),
          (66, 28, 28), (40, 40, 40)]


@pytest.mark.parametrize("gtype", ["r", "d"])
@pytest.mark.parametrize("u8", [True, False])
@pytest.mark.parametrize("shape", LEVELS)
def test_levels_of_thin_volumes(orc, shape, u8, gtype):
    """Whole levels of random images."""
    rng = np.random.default_rng(sum(shape))
    a = rng.random(shape)
    It, Is = (a * 255), (np.clip(a + rng.normal(0, 0.2, shape), 0, 1) * 255)
    It, Is = It.astype(np.uint8 if u8 else np.float32), Is.astype(np.uint8 if u8 else np.float32)
    kw = dict(resolution=1.0, min_dimension=64, gradient_type=gtype)
    d, ok = tb.reg.cdm(It, Is, tb.reg.cdm_param(**kw))
    od, ook, _ = orc.cdm(It, Is, **kw)
    assert ok == ook
    assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
