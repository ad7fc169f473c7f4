"""The Poisson solve (cdm_poisson, reg/cdm.hpp:158-253) of levels small enough for one cluster
a component: 1 to 4 planes a block, the last block partly filled or idle, planes of 1 to 1024
float4 columns, rows that end within a float4 and rows that do not, the first sizes past
each limit, and levels whose sweeps walk 5 to 8 planes a thread -- against the oracle, bit for bit (negative zeros included)."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 5, 4), (2, 1, 1), (15, 7, 9), (16, 8, 8), (17, 6, 5), (31, 9, 12), (32, 16, 20), (33, 5, 7), (46, 31, 33),
          (47, 12, 21), (48, 10, 10), (49, 6, 6), (50, 8, 11), (63, 13, 15), (64, 64, 64), (64, 62, 63), (65, 20, 20),
          (20, 32, 128), (20, 33, 128), (3, 1024, 4), (3, 1025, 3),
          (91, 109, 91), (70, 130, 67), (131, 64, 201)]


@pytest.mark.parametrize("shape", SHAPES)
def test_poisson_clusters(orc, shape):
    rng = np.random.default_rng(sum(shape))
    d = rng.normal(0, 1, shape + (3,)).astype(np.float32)
    d[rng.random(shape) < 0.3] = 0
    d[rng.random(shape) < 0.1] = -0.0
    assert np.array_equal(tb.cdm_poisson(d).view(np.uint32), orc.cdm_poisson(d).view(np.uint32))
