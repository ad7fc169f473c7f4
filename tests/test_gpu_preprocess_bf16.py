"""Preprocessing of BF16 subjects, which the Gaussian reads directly: values of both signs, sizes
where its tiles end, alone and as an engine job -- against the oracle on the widened volume, bit
for bit."""
import numpy as np
import pytest

import tipl_b200 as tb
from tipl_b200 import phantom as ph

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 33), (14, 9, 29), (16, 17, 64), (18, 33, 30), (35, 20, 40), (7, 130, 95)]


@pytest.mark.parametrize("kind", ["both signs", "positive", "negative", "small"])
@pytest.mark.parametrize("shape", SHAPES)
def test_preprocessing_bf16(orc, shape, kind):
    rng = np.random.default_rng(5)
    v = rng.normal(0, 100, shape)
    v = {"both signs": v + 30, "positive": np.abs(v), "negative": -np.abs(v) - 1, "small": np.abs(v) * 1e-6}[kind]
    v[rng.random(shape) < 0.3] = 0
    b = tb.to_bf16(v.astype(np.float32))
    assert np.array_equal(tb.subject_image_pre(b), orc.subject_image_pre(tb.from_bf16(b)))


def test_engine_job_of_a_bf16_subject():
    rng = np.random.default_rng(ph.seed_for(5, 21))
    t = ph.class_phantom((36, 40, 34), rng)
    s = (34, 42, 32)
    T = ph.affine_matrix_f32(ph.random_affine(rng, rot_deg=6, trans_vox=2), s, (1, 1, 1), s, (1, 1, 1))
    m = tb.to_bf16(ph.rician(ph.apply_matrix(ph.class_phantom(s, rng), T, s), rng))
    q_t, _ = tb.normalize_to_u8(t)
    q_m = tb.subject_image_pre(m)
    cost, arg, _ = tb.reg.linear(q_t, (1, 1, 1), q_m, (1, 1, 1))
    Tf = tb.affine_to_matrix(arg, t.shape, (1, 1, 1), m.shape, (1, 1, 1))
    want, ok = tb.reg.cdm(q_t, tb.resample(q_m, t.shape, Tf, allow_shift_copy=True))
    field = np.zeros(t.shape + (3,), np.float32)
    with tb.Engine() as eng:
        tid = eng.add_template(t)
        r = eng.wait(eng.submit(m, template=tid, cdm=True, field_out=field, subject_pre=True))
    assert r["status"] == 0 and r["cdm_ok"] == ok and r["linear_cost"] == np.float32(cost)
    assert np.array_equal(field.view(np.uint32), want.view(np.uint32))
