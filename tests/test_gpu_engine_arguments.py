"""Engine jobs whose CDM parameters cannot be followed are refused when they are submitted."""
import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import _lib

pytestmark = pytest.mark.gpu


def test_min_dimension_zero_is_refused():
    """min_dimension 0 would halve a volume of one voxel for ever; reg.cdm refuses it too."""
    v = np.arange(6 * 5 * 4, dtype=np.uint8).reshape(6, 5, 4)
    p = tb.reg.cdm_param(min_dimension=0)
    with tb.Engine() as eng:
        with pytest.raises(_lib.RegbError) as e:
            eng.submit(v, fixed=v, linear=False, cdm=True, cdm_param=p)
        assert e.value.status == _lib.REGB_ERR_ARG
        assert eng.stats()["queued"] == 0 and eng.stats()["running"] == 0
    with pytest.raises(_lib.RegbError) as e:
        tb.reg.cdm(v, v, p)
    assert e.value.status == _lib.REGB_ERR_ARG
