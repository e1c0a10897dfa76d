"""The float box test's superset property (zt_fast.cuh) out to the farthest
origin it takes: rays from every distance up to kFastMaxOrigin, parallel to
an axis, nearly so, or with components no float holds, against scenes that
are flat, of ordinary size and as large as the records allow.  The limit and
the records' least margin are read from the source, the device arithmetic is
test_fast_slab's restatement."""
import re
from pathlib import Path

import numpy as np
import pytest

from test_fast_slab import f32_slab, f64_slab, out_f32

F32 = np.float32
CSRC = Path(__file__).resolve().parent.parent / "zigtrace_b200" / "csrc"


def _constant(name):
    text = "".join(p.read_text() for p in (CSRC / "zt_fast.cuh", CSRC / "zt_types.h"))
    m = re.search(rf"constexpr \w+ {name} = ([0-9.e+-]+?)f?;", text)
    return float(m[1]) if m else 0.0


def _records(lo, hi, reach):
    eps = np.maximum(np.ldexp(reach, -20), _constant("kFastMinMargin"))
    return out_f32(lo - eps, False), out_f32(hi + eps, True)


# the largest |bound| on each axis
REACH = {"flat": (50.0, 5e-7, 50.0), "thin": (3.0, 3.0, 1e-12), "ordinary": (500.0, 20.0, 500.0),
         "largest": (1e7, 1e7, 1e7)}


@pytest.mark.parametrize("scene", REACH)
def test_superset_from_every_distance_taken(scene):
    rng = np.random.default_rng(len(scene))
    reach = np.array(REACH[scene])
    limit = _constant("kFastMaxOrigin")
    n = 400_000
    mid = rng.uniform(-1, 1, (n, 3)) * reach
    half = 10.0 ** rng.uniform(-6, 0, (n, 3)) * reach
    lo, hi = np.maximum(mid - half, -reach), np.minimum(mid + half, reach)
    lo32, hi32 = _records(lo, hi, reach)
    # a target on the box (corner, edge, face or inside), seen from far away
    u = rng.integers(0, 3, (n, 3))
    tgt = np.where(u == 0, lo, np.where(u == 1, hi, lo + rng.random((n, 3)) * (hi - lo)))
    dist = 10.0 ** rng.uniform(0, np.log10(limit) - 0.3, n)
    d = np.zeros((n, 3))
    ax = rng.integers(0, 3, n)
    rows = np.arange(n)
    d[rows, ax] = rng.choice([-1.0, 1.0], n)
    for k in (1, 2):  # the other components: none, tiny, small
        c = 10.0 ** rng.uniform(-45, 0, n) * rng.choice([-1.0, 0.0, 1.0], n)
        d[rows, (ax + k) % 3] = c
    d /= np.sqrt((d * d).sum(axis=1))[:, None]
    o = tgt - d * dist[:, None]
    taken = np.abs(o.astype(F32)).sum(axis=1, dtype=F32) <= F32(limit)
    with np.errstate(divide="ignore"):
        inv = 1.0 / d
    hits = 0
    for tmin, tmax in ((1e-4, np.inf), (0.0, 2.0 * limit)):
        hit64 = f64_slab(lo, hi, o, inv, tmin, tmax) & taken
        hit32, near32 = f32_slab(lo32, hi32, o, d, tmin, tmax, rcp_ulps=rng.integers(-1, 2, size=(n, 3)))
        missed = hit64 & ~hit32
        assert not missed.any(), f"{missed.sum()} of {hit64.sum()}, nearest {dist[missed].min():.2g}"
        near64 = np.full(n, tmin)
        with np.errstate(invalid="ignore", over="ignore"):
            for a in range(3):
                t = np.where(inv[:, a] < 0, (hi[:, a] - o[:, a]) * inv[:, a], (lo[:, a] - o[:, a]) * inv[:, a])
                near64 = np.where(t > near64, t, near64)
        assert (near32[hit64].astype(np.float64) <= near64[hit64]).all()
        hits += int(hit64.sum())
    assert hits > n // 4
