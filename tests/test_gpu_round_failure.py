"""A round of CDM levels that cannot be run ends the jobs whose levels were in it: each reports
the failure instead of the field its level had reached, and the engine goes on."""
import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import _lib
from tipl_b200 import phantom as ph

pytestmark = pytest.mark.gpu


def test_failed_round_fails_its_jobs():
    """The failure is an allocation made to fail on the host: the first round's status words,
    4 bytes for a round of one level, a size nothing else of such a job asks for."""
    t, m = ph.cdm_class_pair((24, 26, 22), seed=ph.seed_for(5, 401))
    p = tb.reg.cdm_param(resolution=1.0, min_dimension=32)
    want, ok = tb.reg.cdm(t, m, param=p)
    assert ok and np.abs(want).max() > 0
    L = _lib.lib()
    with tb.Engine() as eng:
        assert L.regb_debug_fail_allocations(4, 1) == 0
        try:
            r = eng.wait(eng.submit(m, fixed=t, linear=False, cdm=True, cdm_param=p))
        finally:
            L.regb_debug_fail_allocations(0, 0)
        assert r["status"] == _lib.REGB_ERR_NOMEM
        field = np.zeros(t.shape + (3,), np.float32)
        r = eng.wait(eng.submit(m, fixed=t, linear=False, cdm=True, cdm_param=p, field_out=field))
    assert r["status"] == 0 and r["cdm_ok"]
    assert np.array_equal(field.view(np.uint32), np.asarray(want).view(np.uint32))
