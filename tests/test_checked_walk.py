"""The checked float walk's hit test (walk_reaches, zt_fast.cuh) on the CPU,
the device arithmetic restated in NumPy: wherever it says the f64 walk
reaches a primitive's leaf, the f64 slab test of that primitive's box, and of
larger boxes around it, passes at the hit's distance (aabb.zig:68-83)."""
import numpy as np
import pytest

from test_fast_slab import f64_slab

F32 = np.float32


def walk_reaches(kind, a, o, d, t, reach):
    """kind 1: triangle v0, e1, e2; kind 0: sphere c, r."""
    point = o + d * t[:, None]
    q = (point - a[:, 0:3]).astype(F32)
    slack = (F32(reach) + np.abs(o.astype(F32)).sum(axis=1, dtype=F32)) * F32(2.0 ** -46)
    if kind == 1:
        e1, e2 = a[:, 3:6].astype(F32), a[:, 6:9].astype(F32)
        lo, hi = np.minimum(np.minimum(e1, e2), 0), np.maximum(np.maximum(e1, e2), 0)
        flat = hi - lo < F32(0.99e-6)
        lo, hi = np.where(flat, lo - F32(4.95e-7), lo), np.where(flat, hi + F32(4.95e-7), hi)
    else:
        hi = np.repeat(np.abs(a[:, 3:4]).astype(F32), 3, axis=1)
        lo = -hi
    m = slack[:, None] + np.maximum(-lo, hi) * F32(2.0 ** -20)
    return ((q >= lo + m) & (q <= hi - m)).all(axis=1)


def _targets(rng, n):
    """Barycentrics inside, near edges and on them."""
    u = rng.random((n, 2))
    u = np.where((u.sum(axis=1) > 1)[:, None], 1 - u, u)
    near = 10.0 ** rng.uniform(-17, -4, n)
    u[:, 0] = np.where(rng.random(n) < 0.4, near, u[:, 0])
    u[:, 1] = np.where(rng.random(n) < 0.2, 1 - u[:, 0] - near, u[:, 1])
    return u


def _rays(rng, tgt):
    d = rng.normal(size=tgt.shape)
    par = rng.random(len(d)) < 0.2
    d[par, rng.integers(0, 3, par.sum())] = 0.0
    d /= np.linalg.norm(d, axis=1)[:, None]
    return tgt - d * (10.0 ** rng.uniform(-3, 3.5, len(d)))[:, None], d


@pytest.mark.parametrize("scale", [1.0, 60.0, 3000.0])
@pytest.mark.parametrize("kind", [0, 1])
def test_reached_hits_pass_the_f64_box_test(kind, scale):
    rng = np.random.default_rng(int(scale) + kind)
    n = 200_000
    c = rng.uniform(-scale, scale, (n, 3))
    a = np.zeros((n, 9))
    if kind == 1:
        v = c[:, None, :] + rng.uniform(-0.05, 0.05, (n, 3, 3)) * scale
        flat = rng.random(n) < 0.4  # axis-aligned: the padded box
        ax = rng.integers(0, 3, n)
        v[flat, 1, ax[flat]] = v[flat, 0, ax[flat]]
        v[flat, 2, ax[flat]] = v[flat, 0, ax[flat]]
        a[:, 0:3], a[:, 3:6], a[:, 6:9] = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        lo, hi = v.min(axis=1), v.max(axis=1)
        thin = hi - lo < 1e-6
        lo, hi = np.where(thin, lo - 5e-7, lo), np.where(thin, hi + 5e-7, hi)
        u = _targets(rng, n)
        tgt = a[:, 0:3] + a[:, 3:6] * u[:, :1] + a[:, 6:9] * u[:, 1:]
        o, d = _rays(rng, tgt)
        nrm = np.cross(a[:, 3:6], a[:, 6:9])
        t = ((a[:, 0:3] - o) * nrm).sum(axis=1) / (d * nrm).sum(axis=1)
    else:
        a[:, 0:3], a[:, 3] = c, rng.uniform(0.01, 0.1, n) * scale * np.where(rng.random(n) < 0.2, -1, 1)
        r = np.abs(a[:, 3:4])
        lo, hi = c - r, c + r
        s = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-9, 0, (n, 3))  # many at the poles
        o, d = _rays(rng, c + r * s / np.linalg.norm(s, axis=1)[:, None])
        oc = c - o
        h = (d * oc).sum(axis=1)
        t = h - np.sqrt(np.maximum(h * h - (oc * oc).sum(axis=1) + r[:, 0] ** 2, 0))
    reach = 2 * scale
    with np.errstate(invalid="ignore", divide="ignore"):
        ok = np.isfinite(t) & (t > 1e-4)
        reached = walk_reaches(kind, a, o, d, t, reach) & ok
        inv = 1.0 / d
        # the primitive's box, boxes that share some of its faces, and the root's
        for grow in (0.0, 1e-9, 1.0):
            for side in (0, 1):
                blo = np.maximum(lo - grow * (1 - side), -reach)
                bhi = np.minimum(hi + grow * side, reach)
                passes = f64_slab(blo, bhi, o, inv, 1e-4, t)
                assert (passes | ~reached).all()
    assert reached.mean() > 0.25
