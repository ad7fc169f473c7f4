"""Whole CDM levels where the rows of their component planes meet tiles, padding and odd
forms: widths around multiples of 4, planes smaller and larger than a tile of 512 positions,
rows too short to be padded -- the final fields against the oracle, bit for bit."""
import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import phantom as ph

pytestmark = pytest.mark.gpu


def _pair(shape, u8, seed=3):
    rng = np.random.default_rng(seed)
    c = ph.class_phantom(shape, rng)
    w = ph.rician(ph.warp(c, ph.smooth_field(shape, rng, 6.0, 3.0)), rng)
    return (ph.normalize_to_u8(c), ph.normalize_to_u8(w)) if u8 else (c, w)


@pytest.mark.parametrize("u8", [True, False])
@pytest.mark.parametrize("shape", [(36, 40, 33), (33, 36, 34), (34, 33, 35), (20, 64, 36), (40, 21, 26)])
def test_levels_of_odd_rows(orc, shape, u8):
    It, Is = _pair(shape, u8, ph.seed_for(3, 45))
    d, ok = tb.reg.cdm(It, Is, tb.reg.cdm_param(resolution=1.0))
    od, ook, _ = orc.cdm(It, Is, resolution=1.0)
    assert ok == ook
    assert np.array_equal(d.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("u8", [True, False])
@pytest.mark.parametrize("shape", [(3000, 2, 3), (3, 700, 2), (5, 4, 6)])
def test_levels_of_short_rows(orc, shape, u8):
    """Random images (no phantom fits); one level, since no axis passes min_dimension."""
    rng = np.random.default_rng(7)
    a = rng.random(shape)
    It, Is = (a * 255), (np.clip(a + rng.normal(0, 0.2, shape), 0, 1) * 255)
    It, Is = It.astype(np.uint8 if u8 else np.float32), Is.astype(np.uint8 if u8 else np.float32)
    d, ok = tb.reg.cdm(It, Is, tb.reg.cdm_param(resolution=1.0))
    od, ook, _ = orc.cdm(It, Is, resolution=1.0)
    assert ok == ook
    assert np.array_equal(d.view(np.uint32), od.view(np.uint32))
