"""The checked float walk's certainty about a hit (zt_reach.h, compiled for
the host): sound, since wherever it is certain the f64 box test of the
primitive's box and of boxes around it passes at the hit's distance
(aabb.zig:68-83), also for hits a few roundings from a face and for far
origins; and seldom withheld, also in the middle of a ground made of a large
sphere, where the box touches the sphere."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_checked_walk import _rays, _targets
from test_fast_slab import f64_slab

CSRC = Path(__file__).resolve().parent.parent / "zigtrace_b200" / "csrc"

PROGRAM = """
#include "zt_reach.h"
extern "C" void reaches(long n, int triangle, const double* a, const double* o, const double* p, double reach,
                        unsigned char* out) {
  for (long i = 0; i < n; ++i, a += 9, o += 3, p += 3) {
    const double m = zt::kReachMargin * (reach + fabs(o[0]) + fabs(o[1]) + fabs(o[2]));
    out[i] = zt::reach_inside(triangle != 0, a, p[0] - a[0], p[1] - a[1], p[2] - a[2], m);
  }
}
"""


@pytest.fixture(scope="module")
def reaches(tmp_path_factory):
    d = tmp_path_factory.mktemp("reach")
    (d / "r.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}", "-o",
                    str(d / "r.so"), str(d / "r.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "r.so")).reaches
    ptr = ctypes.c_void_p

    def call(kind, a, o, point, reach):
        a, o, point = (np.ascontiguousarray(x, np.float64) for x in (a, o, point))
        out = np.zeros(len(a), np.uint8)
        fn(ctypes.c_long(len(a)), kind, ptr(a.ctypes.data), ptr(o.ctypes.data), ptr(point.ctypes.data),
           ctypes.c_double(reach), ptr(out.ctypes.data))
        return out != 0
    return call


@pytest.mark.parametrize("scale", [1.0, 60.0, 3000.0, 4e6])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("far", [False, True])
def test_a_certain_hit_passes_the_f64_box_test(reaches, kind, scale, far):
    rng = np.random.default_rng(int(scale) + kind)
    n = 200_000
    c = rng.uniform(-scale, scale, (n, 3))
    a = np.zeros((n, 9))
    if kind == 1:
        v = c[:, None, :] + rng.uniform(-0.05, 0.05, (n, 3, 3)) * scale
        flat = rng.random(n) < 0.5  # axis-aligned, exactly or nearly: the padded box
        ax = rng.integers(0, 3, n)
        for k in (1, 2):
            thick = np.where(rng.random(n) < 0.5, 0.0, 10.0 ** rng.uniform(-9, -5, n)) * rng.choice([-1, 1], n)
            v[flat, k, ax[flat]] = v[flat, 0, ax[flat]] + thick[flat]
        a[:, 0:3], a[:, 3:6], a[:, 6:9] = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        lo, hi = v.min(axis=1), v.max(axis=1)
        thin = hi - lo < 1e-6
        lo, hi = np.where(thin, lo - 5e-7, lo), np.where(thin, hi + 5e-7, hi)
        u = _targets(rng, n)
        tgt = a[:, 0:3] + a[:, 3:6] * u[:, :1] + a[:, 6:9] * u[:, 1:]
    else:
        a[:, 0:3], a[:, 3] = c, rng.uniform(0.01, 0.1, n) * scale * np.where(rng.random(n) < 0.2, -1, 1)
        r = np.abs(a[:, 3:4])
        lo, hi = c - r, c + r
        s = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-9, 0, (n, 3))  # many at the poles
        tgt = c + r * s / np.linalg.norm(s, axis=1)[:, None]
    o, d = _rays(rng, tgt)
    if far:
        o = tgt - d * (10.0 ** rng.uniform(4, 9, n))[:, None]
    if kind == 1:
        nrm = np.cross(a[:, 3:6], a[:, 6:9])
        with np.errstate(invalid="ignore", divide="ignore"):
            t = ((a[:, 0:3] - o) * nrm).sum(axis=1) / (d * nrm).sum(axis=1)
    else:
        oc = c - o
        h = (d * oc).sum(axis=1)
        t = h - np.sqrt(np.maximum(h * h - (oc * oc).sum(axis=1) + r[:, 0] ** 2, 0))
    # half the hits moved to within a few roundings of a face of their box (M + |o| the unit)
    reach = 2 * scale
    unit = (reach + np.abs(o).sum(axis=1)) * 2.0 ** -53
    move = rng.random(n) < 0.5
    axis, up = rng.integers(0, 3, n), rng.random(n) < 0.5
    rows = np.arange(n)
    face = np.where(up, hi[rows, axis], lo[rows, axis])
    inward = np.where(up, -1, 1) * rng.uniform(-4, 80, n) * unit
    with np.errstate(invalid="ignore", divide="ignore", over="ignore"):
        t = np.where(move, (face + inward - o[rows, axis]) / d[rows, axis], t)
        point = o + d * t[:, None]
        certain = reaches(kind, a, o, point, reach) & np.isfinite(t) & (t > 1e-4)
        inv = 1.0 / d
        for grow in (0.0, 1e-9, 1.0):  # the box, boxes that share some of its faces, and the root's
            for side in (0, 1):
                blo = np.maximum(lo - grow * (1 - side), -reach)
                bhi = np.minimum(hi + grow * side, reach)
                assert (f64_slab(blo, bhi, o, inv, 1e-4, t) | ~certain).all()
    assert certain.mean() > 0.02
    assert (certain & move).any()


@pytest.mark.parametrize("radius", [200.0, 1000.0, 5000.0, 1e5])
def test_certain_in_the_middle_of_a_large_sphere(reaches, radius):
    """Hits of camera rays within 12 units of the pole, where a scene stands."""
    rng = np.random.default_rng(int(radius))
    n = 400_000
    x = rng.uniform(-12, 12, (n, 2))
    depth = (x ** 2).sum(axis=1) / (radius + np.sqrt(radius ** 2 - (x ** 2).sum(axis=1)))
    point = np.stack([x[:, 0], -depth, x[:, 1]], axis=1)
    a = np.zeros((n, 9))
    a[:, 1], a[:, 3] = -radius, radius
    o = np.tile([13.0, 2.0, 3.0], (n, 1))
    assert reaches(0, a, o, point, 2 * radius).mean() > 0.9999
