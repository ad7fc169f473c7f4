"""Device memory of a nonlinear registration: what a level holds at once (the high-water mark of
the device's memory pool)."""
import numpy as np
import pytest

import tipl_b200 as tb

pytestmark = pytest.mark.gpu
MB = 1 << 20


def taken(f):
    """The most bytes of the device's memory pool that f holds at once."""
    from cuda.bindings import driver, runtime as rt

    e, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert int(e) == 0
    A = rt.cudaMemPoolAttr

    def get(a):
        e, v = rt.cudaMemPoolGetAttribute(pool, a)
        assert int(e) == 0
        return int(v)

    f()  # what stays with the library is there from now on
    rt.cudaDeviceSynchronize()
    rt.cudaMemPoolSetAttribute(pool, A.cudaMemPoolAttrUsedMemHigh, driver.cuuint64_t(0))
    before = get(A.cudaMemPoolAttrUsedMemCurrent)
    f()
    return get(A.cudaMemPoolAttrUsedMemHigh) - before


def images(shape, dtype=np.uint8):
    rng = np.random.default_rng(11)
    a = rng.random(shape, np.float32) * 200
    return a.astype(dtype), (a + rng.random(shape, np.float32) * 20).astype(dtype)


def level_bytes(shape, px):
    d, h, w = shape
    return 5 * 3 * 4 * (w + 3) // 4 * 4 * h * d + px * w * h * d


# rows that are padded by a third at the level that iterates, and rows that are not padded
@pytest.mark.parametrize("shape", [(1000, 700, 18), (224, 256, 208)])
def test_level_memory(shape):
    """The level that iterates holds five fields and the composed image; its start and its result
    take none beside them."""
    import torch

    It, Is = (torch.from_numpy(v).cuda() for v in images(shape))
    out = torch.zeros(shape + (3,), device="cuda")
    level = tuple((n + 1) // 2 for n in shape)
    p = tb.reg.cdm_param(min_dimension=(min(level) + min(shape)) // 2)
    pyramid = 2 * int(np.prod(level))
    got = taken(lambda: tb.reg.cdm(It, Is, p, out=out))
    assert got <= level_bytes(level, 1) + pyramid + 2 * MB
