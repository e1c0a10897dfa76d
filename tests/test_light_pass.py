"""Lights passed over by the emission pdf (light_passed, zt_device.cuh), the
device arithmetic restated in NumPy: a light passed over adds nothing to
Lights.pdfHit (light.zig:171-198), for points on, beside and away from the
light, small and large lights, near and grazing rays."""
import numpy as np
import pytest

F32 = np.float32


def _out(x, up):
    f = x.astype(F32)
    bad = f.astype(np.float64) < x if up else f.astype(np.float64) > x
    return np.where(bad, np.nextafter(f, F32(np.inf if up else -np.inf)), f)


def _record(v):
    """pass_over_record of scene_host.cpp for triangles v (n, 3, 3)."""
    lo, hi = v.min(axis=1), v.max(axis=1)
    reach = np.maximum(np.abs(lo), np.abs(hi)).max(axis=1)
    e = np.stack([v[:, 1] - v[:, 0], v[:, 2] - v[:, 1], v[:, 0] - v[:, 2]], axis=1)
    length = np.sqrt((e ** 2).sum(axis=2))
    normal = np.cross(e[:, 0], -e[:, 2])
    area = 0.5 * np.sqrt((normal ** 2).sum(axis=1))
    ok = (reach <= 1e7) & (length.max(axis=1) >= 1e-7) & (length[:, 0] * length[:, 2] <= 1e3 * 2 * area)
    pad = (reach * 2.0 ** -21 + 2e-7 * length.max(axis=1))[:, None]
    n = normal / np.maximum(2 * area, 1e-300)[:, None]
    return ok, _out(lo - pad, False), _out(hi + pad, True), n


def _passed(rec, point, to, dist):
    ok, lo, hi, n = rec
    p, t, d = point.astype(F32), to.astype(F32), dist.astype(F32)
    m = (F32(1.2e-6) * d)[:, None]
    outside = ((p + m < lo) | (p - m > hi)).any(axis=1)
    cos = np.abs((t * n.astype(F32)).sum(axis=1, dtype=F32))
    return ok & outside & (cos >= F32(2e-4) * d)


def _contributes(v, o, d, dist):
    """The light's term is reached: triangle.intersect's own f64 steps
    (geometry.zig:83-99), then the distance test."""
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    p = np.cross(d, e2)
    det = (e1 * p).sum(axis=1)
    with np.errstate(all="ignore"):
        inv = 1.0 / det
        s = o - v[:, 0]
        u = (s * p).sum(axis=1) * inv
        q = np.cross(s, e1)
        w = (d * q).sum(axis=1) * inv
        t = (e2 * q).sum(axis=1) * inv
        return (np.abs(det) >= 1e-12) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t > 1e-9) & \
            (np.abs(t - dist) <= 1e-6 * dist)


@pytest.mark.parametrize("size", [1e-3, 1.0, 200.0])
@pytest.mark.parametrize("offset", [0.0, 50.0, 1e5])
def test_a_light_passed_over_adds_nothing(size, offset):
    rng = np.random.default_rng(int(size * 1000 + offset))
    n = 400_000
    c = rng.uniform(-1, 1, (n, 1, 3)) * (offset + 3 * size)
    v = c + rng.uniform(-0.5, 0.5, (n, 3, 3)) * size
    sliver = rng.random(n) < 0.2
    v[sliver, 2] = v[sliver, 0] + (v[sliver, 1] - v[sliver, 0]) * 0.4 + \
        rng.normal(size=(sliver.sum(), 3)) * size * 10.0 ** rng.uniform(-6, -1, (sliver.sum(), 1))
    # a point of the light, moved along and beside the ray by tiny and large amounts
    b = rng.random((n, 2))
    b = np.where((b.sum(axis=1) > 1)[:, None], 1 - b, b)
    b[rng.random(n) < 0.3, 0] = 0.0
    tgt = v[:, 0] + (v[:, 1] - v[:, 0]) * b[:, :1] + (v[:, 2] - v[:, 0]) * b[:, 1:]
    d = rng.normal(size=(n, 3))
    normal = np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    normal /= np.sqrt((normal ** 2).sum(axis=1))[:, None]
    graze = rng.random(n) < 0.4  # rays within 1e-7 .. 1e-2 of the light's plane
    lean = 10.0 ** rng.uniform(-7, -2, n)
    d = np.where(graze[:, None], d - normal * ((d * normal).sum(axis=1) * (1 - lean))[:, None], d)
    d /= np.sqrt((d ** 2).sum(axis=1))[:, None]
    o = tgt - d * (size * 10.0 ** rng.uniform(-2, 3, n))[:, None]
    move = np.where(rng.random(n) < 0.5, 0.0, 10.0 ** rng.uniform(-9, 0, n)) * rng.choice([-1, 1], n)
    point = tgt + d * (move * size)[:, None]
    to = point - o
    dist = np.sqrt((to ** 2).sum(axis=1))
    ok = dist > 1e-9
    dirs = to * (1 / np.where(ok, dist, 1))[:, None]
    passed = _passed(_record(v), point, to, dist) & ok
    contributes = _contributes(v, o, dirs, dist) & ok
    assert not (passed & contributes).any()
    assert contributes.mean() > 0.2
    if size < 2.0 ** -18 * (offset + 3 * size):  # smaller than single precision resolves there: none is passed over
        return
    # and it does pass lights over: points well away from them
    far = point + size * (2 + rng.random((n, 1))) * rng.choice([-1.0, 1.0], (n, 3))
    to = far - o
    assert (_passed(_record(v), far, to, np.sqrt((to ** 2).sum(axis=1))) | sliver).mean() > 0.5
