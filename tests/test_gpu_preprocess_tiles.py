"""subject_image_pre (reg/mm_reg.hpp:14-20) and the Gaussian where tiles end: widths around 32
columns, heights around the 4 rows of a warp and 16 of a block, depths around 15 planes, every
storage type, counts above the threshold on both sides of the chunked median's 2048, flat,
two-valued and negative images, an output at an odd address -- against the oracle, bit for
bit."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 1, 33), (2, 5, 32), (14, 9, 29), (15, 16, 31), (16, 17, 64), (17, 3, 65), (18, 33, 30), (35, 20, 40),
          (7, 130, 95)]


@pytest.mark.parametrize("shape", SHAPES)
def test_gaussian_tiles(orc, shape):
    v = np.random.default_rng(1).normal(0, 100, shape).astype(np.float32)
    for rounds in (1, 2, 3):
        assert np.array_equal(tb.gaussian(v, rounds).view(np.uint32), orc.gaussian(v, rounds).view(np.uint32))


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_preprocessing_tiles(orc, shape, dtype):
    rng = np.random.default_rng(2)
    v = (rng.random(shape) * (250 if dtype == np.uint8 else 3000)).astype(dtype)
    v[rng.random(shape) < 0.5] = 0
    assert np.array_equal(tb.subject_image_pre(v), orc.subject_image_pre(v.astype(np.float32)))


@pytest.mark.parametrize("kind", ["flat", "zero", "two", "negative", "narrow", "wide"])
def test_preprocessing_values(orc, kind):
    rng = np.random.default_rng(3)
    n = rng.normal(0, 1, (24, 30, 34)).astype(np.float32)
    v = {"flat": np.full_like(n, 7.0), "zero": np.zeros_like(n), "two": np.where(n > 0.8, 5.0, 1.0),
         "negative": n - 50.0, "narrow": 1000.0 + n * 1e-3, "wide": np.exp(8.0 * n)}[kind].astype(np.float32)
    assert np.array_equal(tb.subject_image_pre(v), orc.subject_image_pre(v))


def test_preprocessing_into_any_address(orc):
    import torch

    v = (np.random.default_rng(4).random((20, 21, 23)) * 900).astype(np.uint16)
    ref = orc.subject_image_pre(v.astype(np.float32))
    for off in (1, 2, 4):
        buf = torch.zeros(v.size + off, dtype=torch.uint8, device="cuda")
        tb.subject_image_pre(torch.from_numpy(v).cuda(), out=buf[off:].view(v.shape))
        assert np.array_equal(buf[off:].cpu().numpy().reshape(v.shape), ref)
