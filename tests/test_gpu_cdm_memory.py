"""Device memory of a nonlinear registration: what a level holds, and the engine's estimate of a
job against what the job takes from the device's memory pool (its high-water mark)."""
import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import _lib

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


CASES = {
    "u8": dict(shape=(1000, 700, 18), dtype=np.uint8),
    "f32": dict(shape=(600, 700, 18), dtype=np.float32),
    "mm_reg": dict(shape=(700, 600, 18), dtype=np.uint16, mm=True),
    "one level": dict(shape=(500, 700, 9), dtype=np.float32, resolution=1.0),
}


@pytest.mark.parametrize("name", CASES)
def test_engine_estimate_covers_a_job(name):
    """An engine whose budget is a byte less than what the job takes refuses it."""
    c = CASES[name]
    fixed, moving = images(c["shape"], c["dtype"])
    mm = c.get("mm", False)
    kw = dict(fixed=fixed, linear=mm, cdm=True, subject_pre=mm, mm_reg=mm,
              cdm_param=tb.reg.cdm_param(resolution=c.get("resolution", 2.0)))
    with tb.Engine() as eng:
        def job():
            assert eng.wait(eng.submit(moving, **kw))["status"] == 0

        need = taken(job)
    with tb.Engine(hbm_budget_bytes=need - 1) as eng:
        with pytest.raises(_lib.RegbError) as e:
            eng.submit(moving, **kw)
        assert e.value.status == _lib.REGB_ERR_BUDGET


def test_engine_admits_preprocessing_that_fits():
    """The estimate of a job that only preprocesses counts the buffers it has: its volume, the
    result, two float copies, and the 16 MB that every estimate has on top."""
    v = images((128, 256, 160), np.uint16)[1]
    kw = dict(fixed=v[:8, :8, :8].copy(), linear=False, subject_pre=True)
    with tb.Engine() as eng:
        need = taken(lambda: eng.wait(eng.submit(v, **kw)))
    with tb.Engine(hbm_budget_bytes=need + 17 * MB) as eng:
        assert eng.wait(eng.submit(v, **kw))["status"] == 0
