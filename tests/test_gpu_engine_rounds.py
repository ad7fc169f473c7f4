"""Rounds that several CDM levels share, of every form a level's passes take: sweeps in clusters,
walked planes, a component in one line, rows without padding; gradients in tiles and a voxel a
thread.  Jobs join while others run, and each field is the plain call's, bit for bit."""
import time

import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import phantom as ph

pytestmark = pytest.mark.gpu

# too large for the clusters (two of them walk their planes), then small, flat and long ones
SHAPES = [(70, 66, 68), (40, 80, 66), (66, 40, 84), (26, 30, 24), (64, 20, 33), (70, 8, 8), (66, 60, 2), (3, 120, 120),
          (100, 100, 3), (2, 90, 70)]


def _pair(shape, seed):
    if min(shape) >= 20:
        return ph.cdm_class_pair(shape, seed=seed)
    rng = np.random.default_rng(seed)
    a = rng.random(shape) * 255
    return a.astype(np.float32), np.clip(a + rng.normal(0, 20, shape), 0, 255).astype(np.float32)


@pytest.mark.parametrize("gap_ms", [0.0, 0.7])
@pytest.mark.parametrize("u8", [False, True])
def test_mixed_rounds_equal_plain(u8, gap_ms):
    p = tb.reg.cdm_param(resolution=1.0, min_dimension=128)
    cases = []
    for k in range(2 * len(SHAPES)):
        t, m = _pair(SHAPES[k % len(SHAPES)], ph.seed_for(5, 500 + k))
        cases.append(tuple(ph.normalize_to_u8(v) for v in (t, m)) if u8 else (t, m))
    want = [tb.reg.cdm(t, m, param=p) for t, m in cases]
    outs = [np.zeros(t.shape + (3,), np.float32) for t, _ in cases]
    with tb.Engine(max_active=64) as eng:
        ids = []
        for (t, m), o in zip(cases, outs):
            ids.append(eng.submit(m, fixed=t, linear=False, cdm=True, cdm_param=p, field_out=o))
            time.sleep(gap_ms * 1e-3)
        res = [eng.wait(i) for i in ids]
        st = eng.stats()
    for (f, ok), o, r in zip(want, outs, res):
        assert r["status"] == 0 and bool(r["cdm_ok"]) == bool(ok)
        assert np.array_equal(np.asarray(f, np.float32).view(np.uint32), o.view(np.uint32))
    # (thin volumes end without a field: their edges leave the volume with any)
    assert all(float(np.abs(o).max()) > 0.1 for (t, _), o in zip(cases, outs) if min(t.shape) >= 40)
    assert st["cdm_max_round_segments"] >= 4
