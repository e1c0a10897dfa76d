"""zt_scene_upload_bytes counts what the device copy of a scene holds: no
float records where a leaf of the tree is too large for them (15 primitives,
FPair in zt_types.h), and the same number before, between and after
uploads."""
import numpy as np
import pytest

import zigtrace_b200 as zt
from zigtrace_b200 import _native as N


def two_leaves(left, n=30):
    """n spheres under a root with leaves of `left` and n - left."""
    rng = np.random.default_rng(n)
    c = np.stack([np.arange(n, dtype=float), rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)], axis=1)
    s = zt.Scene()
    s.background = zt.Background.sky((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    s.add_spheres(c, np.full(n, 0.4), s.add_material(zt.Material.lambertian((0.4, 0.5, 0.6))))
    s.camera = zt.CameraConfig(look_from=(n / 2, 0.0, 30.0), look_at=(n / 2, 0.0, 0.0))
    nodes = np.zeros(3, N.BVH_NODE_DTYPE)
    for i, (a, b) in enumerate(((0, n), (0, left), (left, n))):
        nodes["bmin"][i], nodes["bmax"][i] = c[a:b].min(axis=0) - 0.4, c[a:b].max(axis=0) + 0.4
        nodes["first"][i], nodes["count"][i] = a, b - a
    nodes["first"][0], nodes["count"][0] = 1, 0
    return s.build_with_bvh(nodes, np.arange(n, dtype=np.uint32))


def test_no_float_records_for_a_large_leaf():
    assert two_leaves(15).staging_bytes() - two_leaves(16).staging_bytes() == 256  # one record, in a block of its own


@pytest.mark.gpu
@pytest.mark.parametrize("left", [15, 16])
def test_the_same_before_and_after_uploads(left):
    s = two_leaves(left)
    want = s.staging_bytes()
    o = zt.Options(48, 32, 4, 6, seed=2)
    images = set()
    for _ in range(3):
        s.upload()
        assert s.staging_bytes() == want
        for precision in (zt.PRECISION_EXACT, zt.PRECISION_FAST):
            images.add(zt.render(s, o, zt.GpuConfig(precision=precision)).pixels.tobytes())
        s.release_device()
        assert s.staging_bytes() == want
    images.add(zt.render(s, o, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels.tobytes())
    assert len(images) == 1
