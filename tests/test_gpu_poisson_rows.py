"""The Poisson solve (cdm_poisson, reg/cdm.hpp:158-253) where rows, planes and padding meet:
widths around multiples of 4, planes smaller than a block, single rows and planes, more
planes than a thread walks, and rows too short to be padded -- against the oracle, bit for
bit (negative zeros included)."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 2), (2, 3, 1), (3, 2, 3), (1, 9, 4), (5, 4, 5), (7, 1, 40), (9, 26, 36), (17, 27, 37),
          (8, 25, 38), (2, 33, 31), (16, 40, 129), (23, 28, 23), (64, 64, 64), (3, 700, 2), (2, 2, 1500),
          (2100, 2000, 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_poisson_rows(orc, shape):
    rng = np.random.default_rng(sum(shape))
    d = rng.normal(0, 1, shape + (3,)).astype(np.float32)
    d[rng.random(shape) < 0.3] = 0
    d[rng.random(shape) < 0.1] = -0.0
    assert np.array_equal(tb.cdm_poisson(d).view(np.uint32), orc.cdm_poisson(d).view(np.uint32))
