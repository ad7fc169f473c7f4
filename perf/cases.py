"""Timed cases of the registration path: what a user of tipl_b200 has it do, through the
public calls, over the range of sizes and types they are made with.

A case is a dict of plain values; ``op`` names the call.  Sizes are (x, y, z) voxels: the
64^3, 128^3 and 182x218x182 grids of the package's templates, the 2 mm 91x109x91 grid, the
96 to 256 voxel sides of subject scans, and odd sizes between them.  Volumes are the seeded
class phantoms of tipl_b200.phantom (three intensity classes in a smoothed ellipsoid, 2 %
Rician noise, a smooth warp of up to 4 voxels or a random affine), made here with torch on
the device.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tipl_b200 as tb
from tipl_b200 import phantom as ph

DEV = "cuda"
ONE = (1.0, 1.0, 1.0)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one optimiser probe of a coarse pyramid level: the smallest call, all latency
        {"name": "mi_cost_64_k1", "op": "mi_cost", "x": 64, "y": 64, "z": 64, "k": 1},
        # a line-search probe set at the template's own resolution
        {"name": "mi_cost_182_k16", "op": "mi_cost", "x": 182, "y": 218, "z": 182, "k": 16},
        # the correlation cost's probe set on a large subject scan
        {"name": "corr_cost_256_k8", "op": "corr_cost", "x": 256, "y": 256, "z": 200, "k": 8},
        # subject preprocessing of a large uint16 scan before its registration
        {"name": "pre_u16_256", "op": "pre", "x": 256, "y": 256, "z": 200, "dtype": "u16"},
        # the local-correlation gradient of the float path on an odd-sized volume
        {"name": "gradient_f32_157", "op": "gradient", "x": 157, "y": 189, "z": 155, "dtype": "f32"},
        # the Poisson solve of a full-resolution update field
        {"name": "poisson_182", "op": "poisson", "x": 182, "y": 218, "z": 182},
        # a whole nonlinear registration of a small float pair, default parameters
        {"name": "cdm_f32_64", "op": "cdm", "x": 64, "y": 64, "z": 64, "dtype": "f32", "resolution": 2.0,
         "min_dimension": 16},
        # the uint8 nonlinear registration to the 1 mm template (mm_reg's stage)
        {"name": "cdm_u8_182", "op": "cdm", "x": 182, "y": 218, "z": 182, "dtype": "u8", "resolution": 2.0,
         "min_dimension": 32},
        # a float pair iterated at its full resolution: the largest fields
        {"name": "cdm_f32_128_full", "op": "cdm", "x": 128, "y": 128, "z": 128, "dtype": "f32", "resolution": 1.0,
         "min_dimension": 32},
        # the affine search with mutual information at 1 mm
        {"name": "linear_mi_182", "op": "linear", "x": 182, "y": 218, "z": 182, "cost": "mi"},
        # eight uneven uint16 subjects served at once: affine MI, then float CDM
        {"name": "engine_u16_x8", "op": "engine", "x": 182, "y": 218, "z": 182, "jobs": 8, "side_lo": 96,
         "side_hi": 192, "mm_reg": False},
        # the mm_reg pipeline of two subjects: preprocessing, correlation affine, uint8 CDM both ways
        {"name": "engine_mm_reg_x2", "op": "engine", "x": 128, "y": 128, "z": 128, "jobs": 2, "side_lo": 112,
         "side_hi": 160, "mm_reg": True},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["mi_cost", "corr_cost", "pre", "gradient", "poisson", "cdm", "cdm", "linear", "engine"])
    if op in ("mi_cost", "corr_cost"):
        c = {"op": op, "k": rng.choice([1, 2, 3, 5, 8, 12, 16])}
        c.update({a: _side(rng, 48, 200) for a in "xyz"})
        return c
    if op == "pre":
        c = {"op": op, "dtype": rng.choice(["u16", "f32"])}
        c.update({a: _side(rng, 64, 220) for a in "xyz"})
        return c
    if op in ("gradient", "poisson"):
        c = {"op": op}
        if op == "gradient":
            c["dtype"] = rng.choice(["u8", "f32"])
        c.update({a: _side(rng, 24, 200) for a in "xyz"})
        return c
    if op == "cdm":
        full = rng.random() < 0.5
        c = {"op": op, "dtype": rng.choice(["u8", "f32"]), "resolution": 1.0 if full else 2.0,
             "min_dimension": rng.choice([16, 32])}
        c.update({a: _side(rng, 48, 112 if full else 182) for a in "xyz"})
        return c
    if op == "linear":
        c = {"op": op, "cost": rng.choice(["mi", "corr"])}
        c.update({a: _side(rng, 64, 182) for a in "xyz"})
        return c
    mm = rng.random() < 0.4
    t = rng.choice([(64, 64, 64), (91, 109, 91), (128, 128, 128)])
    lo = rng.randint(72, 104)
    return {"op": op, "x": t[0], "y": t[1], "z": t[2], "jobs": rng.randint(1, 2 if mm else 5), "side_lo": lo,
            "side_hi": lo + rng.randint(16, 48), "mm_reg": mm}


# ---------------------------------------------------------------- volumes, on the device
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _band(n, sigma):
    """Gaussian smoothing along an axis of n samples as a matrix (rows sum to 1)."""
    i = torch.arange(n, dtype=torch.float32, device=DEV)
    m = torch.exp(-((i[:, None] - i[None, :]) ** 2) / (2 * sigma * sigma))
    return m / m.sum(1, keepdim=True)


def _smooth(v, sigma):
    d, h, w = v.shape
    v = (_band(d, sigma) @ v.reshape(d, h * w)).reshape(d, h, w)
    v = torch.matmul(_band(h, sigma), v)
    return torch.matmul(v, _band(w, sigma).t())


def _axes(shape):
    return [torch.arange(n, dtype=torch.float32, device=DEV) for n in shape]


def _phantom(shape, rng, g):
    """The class phantom: 0 outside a smoothed ellipsoid, two intensity levels inside, with the
    1 % texture that an averaged template has."""
    z, y, x = _axes(shape)
    d2 = []
    for ax, n in zip((z, y, x), shape):
        c = torch.tensor(rng.uniform(0, n, 32), dtype=torch.float32, device=DEV)
        d2.append((ax[None, :] - c[:, None]) ** 2)
    s = torch.tensor(rng.uniform(3.0, 8.0, 32) * max(1.0, min(shape) / 96.0), dtype=torch.float32, device=DEV)
    a = torch.tensor(rng.uniform(0.2, 1.0, 32), dtype=torch.float32, device=DEV)
    e = [torch.exp(-q / (2 * s * s)[:, None]) for q in d2]
    blobs = ((e[0] * a[:, None]).t() @ (e[1][:, :, None] * e[2][:, None, :]).reshape(32, -1)).reshape(shape)
    blobs = blobs / blobs.max().clamp_min(1e-6)
    q = sum(((ax - (n - 1) / 2.0) / (0.42 * n)).square().reshape([-1 if i == j else 1 for j in range(3)])
            for i, (ax, n) in enumerate(zip((z, y, x), shape)))
    mask = _smooth((q <= 1.0).float(), 2.0)
    mask = torch.where(mask < 1e-3, torch.zeros_like(mask), mask)  # the background is exactly 0
    lo, hi = rng.uniform(800, 1200), rng.uniform(2500, 3200)
    t = ((blobs - 0.35) / 0.2).clamp(0.0, 1.0)
    texture = 1.0 + 0.01 * torch.randn(shape, generator=g, device=DEV)
    return (mask * (lo + (hi - lo) * t) * texture).clamp(0, 4095)


def _sample(v, px, py, pz):
    """trilinear(v, p), 0 where the cell leaves the volume."""
    d, h, w = v.shape
    ok = (px >= 0) & (py >= 0) & (pz >= 0) & (px < w - 1) & (py < h - 1) & (pz < d - 1)
    ix, iy, iz = (torch.where(ok, p, torch.zeros_like(p)).floor().long() for p in (px, py, pz))
    fx, fy, fz = px - ix, py - iy, pz - iz
    f = v.reshape(-1)
    out = torch.zeros_like(px)
    for k in range(8):
        i, j, m = k & 1, (k >> 1) & 1, k >> 2
        wt = (fx if i else 1 - fx) * (fy if j else 1 - fy) * (fz if m else 1 - fz)
        out = out + wt * f[((iz + m) * h + iy + j) * w + ix + i].to(px.dtype)
    return torch.where(ok, out, torch.zeros_like(out))


def _rician(v, g):
    s = 0.02 * float(v.max())
    a = v + s * torch.randn(v.shape, generator=g, device=DEV)
    b = s * torch.randn(v.shape, generator=g, device=DEV)
    return torch.sqrt(a * a + b * b)


def _grid(shape):
    z, y, x = _axes(shape)
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _warped(v, g, max_len):
    """v under a smooth displacement (white noise smoothed with sigma 6, up to max_len voxels)."""
    d = torch.stack([_smooth(torch.randn(v.shape, generator=g, device=DEV), 6.0) for _ in range(3)])
    d = d * (max_len / d.square().sum(0).sqrt().max())
    x, y, z = _grid(v.shape)
    return _rician(_sample(v, x + d[0], y + d[1], z + d[2]), g)


def _moved(v, T, shape, g):
    """v under the voxel transform T on a grid of the given shape."""
    x, y, z = _grid(shape)
    T = [float(t) for t in T]
    p = [T[3 * a] * x + T[3 * a + 1] * y + T[3 * a + 2] * z + T[9 + a] for a in range(3)]
    return _rician(_sample(v, *p), g)


def _u8(v):
    lo, hi = v.min(), v.max()
    return ((v - lo) * (255.999 / (hi - lo))).to(torch.uint8)


def _typed(v, dtype):
    if dtype == "u8":
        return _u8(v)
    if dtype == "u16":
        return v.clamp(0, 4095).to(torch.int32).to(torch.uint16)
    return v.contiguous()


def _shape(case):
    return (int(case["z"]), int(case["y"]), int(case["x"]))


def _subject(t, shape, vs, rng, g):
    """A subject made from the 1 mm template t by a random affine, on a grid of its own (float)."""
    p = ph.random_affine(rng, trans_vox=min(10.0, min(t.shape) / 16.0))
    return _moved(t, ph.affine_matrix_f32(p, shape, (vs,) * 3, tuple(t.shape), ONE), shape, g)


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    rng, g, op = np.random.default_rng(seed), _gen(seed), case["op"]
    shape = _shape(case)
    if op in ("mi_cost", "corr_cost"):
        t = _phantom(shape, rng, g)
        m = _subject(t, shape, 1.0, rng, g)
        # a probe set: small steps around a nearby transform
        Ts = []
        for _ in range(int(case["k"])):
            q = ph.random_affine(rng, rot_deg=4.0, trans_vox=3.0, scale=(0.96, 1.04), shear=0.02)
            Ts.append(tb.affine_to_matrix(q, shape, ONE, shape, ONE))
        return {"op": op, "f": _u8(t), "m": _u8(m), "T": np.array(Ts, np.float32)}
    if op == "pre":
        v = _typed(_rician(_phantom(shape, rng, g), g), case["dtype"])
        return {"op": op, "v": v, "out": torch.zeros(shape, dtype=torch.uint8, device=DEV)}
    if op == "gradient":
        t = _phantom(shape, rng, g)
        return {"op": op, "It": _typed(t, case["dtype"]), "Js": _typed(_warped(t, g, 3.0), case["dtype"])}
    if op == "poisson":
        # an update field: large on the object, 0 on the background, as the gradient leaves it
        t = _phantom(shape, rng, g)
        d = torch.randn(shape + (3,), generator=g, device=DEV) * t[..., None] * (t[..., None] > 0)
        return {"op": op, "d": d.contiguous()}
    if op == "cdm":
        t = _phantom(shape, rng, g)
        m = _warped(t, g, 3.0 if min(shape) < 96 else 4.0)
        return {"op": op, "It": _typed(t, case["dtype"]), "Is": _typed(m, case["dtype"]),
                "par": tb.reg.cdm_param(resolution=float(case["resolution"]),
                                        min_dimension=int(case["min_dimension"])),
                "out": torch.zeros(shape + (3,), dtype=torch.float32, device=DEV)}
    if op == "linear":
        t = _phantom(shape, rng, g)
        m = _subject(t, shape, 1.0, rng, g)
        cost = tb.reg.MI if case["cost"] == "mi" else tb.reg.CORR
        return {"op": op, "f": _u8(t), "m": _u8(m), "par": tb.reg.linear_param(cost_type=cost)}
    # engine: one resident template, the subjects that come in
    mm = bool(case["mm_reg"])
    t = _phantom(shape, rng, g)
    e = tb.Engine()
    tid = e.add_template(_typed(t, "u8" if mm else "u16"), ONE)
    subjects, outs = [], []
    lo, hi, jobs = (int(case[k]) for k in ("side_lo", "side_hi", "jobs"))
    shapes = np.random.default_rng([lo, hi, jobs]).integers(lo, hi + 1, (jobs, 3))  # uneven, the case's own
    for ss in shapes:
        ss = tuple(int(v) for v in ss)
        vs = round(max(shape) / (1.1 * min(ss)), 3)  # the subject's field of view covers the template
        subjects.append((_typed(_subject(t, ss, vs, rng, g), "u16"), (vs,) * 3))
        o = {"field_out": torch.zeros(shape + (3,), dtype=torch.float32, device=DEV)}
        if mm:
            o["field_rev_out"] = torch.zeros_like(o["field_out"])
            o["mapping_out"] = torch.zeros_like(o["field_out"])
            o["inv_mapping_out"] = torch.zeros(ss + (3,), dtype=torch.float32, device=DEV)
        outs.append(o)
    return {"op": op, "engine": e, "tid": tid, "subjects": subjects, "outs": outs, "mm": mm,
            "par": tb.reg.cdm_param(min_dimension=32)}


def run(s):
    op = s["op"]
    if op == "mi_cost":
        return tb.mi_cost(s["f"], s["m"], s["T"])
    if op == "corr_cost":
        return tb.corr_cost(s["f"], s["m"], s["T"])
    if op == "pre":
        return tb.subject_image_pre(s["v"], out=s["out"])
    if op == "gradient":
        return tb.cdm_gradient(s["Js"], s["It"])
    if op == "poisson":
        return tb.cdm_poisson(s["d"])
    if op == "cdm":
        return tb.reg.cdm(s["It"], s["Is"], s["par"], out=s["out"])
    if op == "linear":
        return tb.reg.linear(s["f"], ONE, s["m"], ONE, param=s["par"])
    e = s["engine"]
    ids = [e.submit(v, vs, template=s["tid"], cdm=True, cdm_param=s["par"], subject_pre=s["mm"], mm_reg=s["mm"], **o)
           for (v, vs), o in zip(s["subjects"], s["outs"])]
    res = [e.wait(i) for i in ids]
    keys = ("status", "linear_cost", "arg", "cost_evals", "cdm_ok", "cdm_iterations")
    keys += ("cdm_rev_ok", "r_linear", "r_nonlinear") if s["mm"] else ()
    # a result's scalars in one array beside the job's fields
    return [{"result": np.concatenate([np.ravel(np.asarray(r[k], np.float64)) for k in keys]), **o}
            for r, o in zip(res, s["outs"])]


# ---------------------------------------------------------------- the work a pass cannot do without
# Arithmetic of a voxel: a trilinear sample with its transform ~40, a cost's counts ~4; a CDM
# iteration ~40 (warp) + 5 window sums (separable, 5 x 3 x 4) and the regression ~100 + 12
# sweeps x 3 components x 7 + ~110 (composition) + 3 x 8 (smoothing).
SAMPLE = 44
CDM_ITER = 40 + 100 + 12 * 21 + 110 + 24
# How often the loops run is the data's; these are ordinary counts, for the scale only.
MI_EVALS, CDM_ITERS = 2300, 60


def _linear_work(n, m):
    # the pyramid halves while a level holds more than 96^3 voxels: about a fifth of the
    # evaluations at full resolution
    evals = MI_EVALS * (0.25 if n > 96 ** 3 else 1.0)
    return {"bytes": n + m, "flops": evals * n * SAMPLE}


def _cdm_work(n, psz, resolution):
    it = n if resolution <= 1.0 else n / 8.0
    return {"bytes": 2 * n * psz + 12 * n, "flops": CDM_ITERS * it * CDM_ITER}


def work(case):
    n, op = math.prod(_shape(case)), case["op"]
    psz = {"u8": 1, "u16": 2, "f32": 4}.get(case.get("dtype"), 1)
    if op in ("mi_cost", "corr_cost"):
        k = int(case["k"])
        return {"bytes": 2 * n + 56 * k, "flops": k * n * SAMPLE}
    if op == "pre":
        return {"bytes": n * (psz + 1), "flops": n * 40}
    if op == "gradient":
        return {"bytes": n * (2 * psz + 12), "flops": n * 100}
    if op == "poisson":
        return {"bytes": n * 24, "flops": n * 12 * 21}
    if op == "cdm":
        return _cdm_work(n, psz, float(case["resolution"]))
    if op == "linear":
        return _linear_work(n, n)
    m = (0.5 * (case["side_lo"] + case["side_hi"])) ** 3
    mm = bool(case["mm_reg"])
    a, b = _linear_work(n, m), _cdm_work(n, 1 if mm else 4, 2.0)
    jobs, ways = int(case["jobs"]), 2 if mm else 1
    out = jobs * (24 * n + 12 * m) if mm else 0
    return {"bytes": jobs * (n + 2 * m + 12 * n) + out, "flops": jobs * (a["flops"] + ways * b["flops"])}


# ---------------------------------------------------------------- 64-bit values
def _exact_cost(s):
    f, m = s["f"], s["m"]
    x, y, z = (v.double() for v in _grid(f.shape))
    out = []
    for T in s["T"].astype(np.float64):
        p = [T[3 * a] * x + T[3 * a + 1] * y + T[3 * a + 2] * z + T[9 + a] for a in range(3)]
        v = _sample(m, *p).floor().clamp(0, 255)
        if s["op"] == "corr_cost":
            a, b = f.double(), v
            a, b = a - a.mean(), b - b.mean()
            r = float((a * b).mean() / (a.square().mean().sqrt() * b.square().mean().sqrt()))
            out.append(1.0 - r * r)
            continue
        h = torch.bincount((f.long() * 256 + v.long()).reshape(-1), minlength=65536).double().reshape(256, 256)
        rc = h.sum(1, keepdim=True) * h.sum(0, keepdim=True)
        # -sum mu ln(mu / row / col) / 65536 with the counts themselves
        t = torch.where(h > 0, h * (h.clamp_min(1.0).log() - rc.clamp_min(1.0).log()), torch.zeros_like(h))
        out.append(-float(t.sum()) / 65536.0)
    return np.array(out, np.float64)


def _box5(v):
    """Sums over the 5^3 window clipped to the volume."""
    for a in range(3):
        pad = [0, 0, 0, 0, 0, 0]
        pad[2 * (2 - a)] = pad[2 * (2 - a) + 1] = 2
        q = torch.nn.functional.pad(v, pad)
        v = sum(q.narrow(a, k, v.shape[a]) for k in range(5))
    return v


def _exact_gradient(s):
    j, t = s["Js"].double(), s["It"].double()
    n = _box5(torch.ones_like(j))
    mx, my = _box5(j) / n, _box5(t) / n
    xv, yv = _box5(j * j) / n - mx * mx, _box5(t * t) / n - my * my
    cov = _box5(j * t) / n - mx * my
    ok = (j != 0) & (t != 0) & (xv > 0) & (yv > 0) & (cov > 0)
    xv, yv = torch.where(ok, xv, torch.ones_like(xv)), torch.where(ok, yv, torch.ones_like(yv))
    a, r2 = cov / xv, cov * cov / xv / yv
    k = torch.where(ok, r2 * (j * a + my - a * mx - t), torch.zeros_like(j))
    g = torch.zeros(j.shape + (3,), dtype=torch.float64, device=j.device)
    g[:, :, 1:-1, 0] = j[:, :, 2:] - j[:, :, :-2]
    g[:, 1:-1, :, 1] = j[:, 2:] - j[:, :-2]
    g[1:-1, :, :, 2] = j[2:] - j[:-2]
    return g * k[..., None], -float(torch.where(ok, r2, torch.zeros_like(r2)).mean())


def _exact_poisson(s):
    # the sweeps take their neighbours by flat index
    d = s["d"].double()
    h, w = d.shape[1:3]
    r = d.reshape(-1, 3)
    v = r * (-1.0 / 6.0)
    for _ in range(12):
        q = r.clone()
        for k in (1, w, w * h):
            q[k:] -= v[:-k]
            q[:-k] -= v[k:]
        v = q * (-1.0 / 6.0)
    return v.reshape(d.shape)


def exact(case, seed):
    op = case["op"]
    if op in ("mi_cost", "corr_cost"):
        return _exact_cost(prepare(case, seed))
    if op == "gradient":
        return _exact_gradient(prepare(case, seed))
    if op == "poisson":
        return _exact_poisson(prepare(case, seed))
    return None  # bytes, or loops whose length the data decides
