"""Scenes flattened on the device: from a device build, from a host build, released and uploaded again (from the device, then from
the pinned image), imported with leaves too large for the float records, and
with a NaN -- every mode bit-identical to the oracle's image of the scene."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu

N = 16400
OPTS = zt.Options(40, 28, 3, 8, seed=6)
CONFIGS = [zt.GpuConfig(zt.MODE_MEGAKERNEL), zt.GpuConfig(zt.MODE_WAVEFRONT),
           zt.GpuConfig(zt.MODE_MEGAKERNEL_REGEN, precision=zt.PRECISION_FAST)]


def mixed(n=N, seed=1):
    rng = np.random.default_rng(seed)
    s = zt.Scene()
    mats = [s.add_material(zt.Material.lambertian(rng.uniform(0.2, 0.9, 3))),
            s.add_material(zt.Material.metal(rng.uniform(0.4, 1.0, 3), 0.2)),
            s.add_material(zt.Material.dielectric(1.5)),
            s.add_material(zt.Material.emissive((4.0, 3.0, 2.0)))]
    s.add(zt.plane((0, -6, 0), (0, 1, 0), mats[0]))
    k = n // 2
    s.add_spheres(rng.uniform(-5, 5, (k, 3)), rng.uniform(0.02, 0.08, k) * rng.choice([1, 1, -1], k),
                  rng.choice(mats[:3], k))
    c = rng.uniform(-5, 5, (n - k, 3))
    s.add_triangles(c, c + rng.uniform(-.2, .2, c.shape), c + rng.uniform(-.2, .2, c.shape),
                    np.where(rng.random(n - k) < 0.01, mats[3], mats[0]))
    s.camera = zt.CameraConfig(look_from=(0, 1, 14), look_at=(0, 0, 0), vfov=45)
    return s


@pytest.fixture(scope="module")
def want():
    return O.OracleScene.from_scene(mixed()).render(OPTS.width, OPTS.height, OPTS.spp, OPTS.max_depth, seed=OPTS.seed)


def _check(scene, want):
    for cfg in CONFIGS:
        img = zt.render(scene, OPTS, cfg).pixels
        same = (img == want).all(axis=1).mean()
        assert same == 1.0 if cfg.precision == zt.PRECISION_EXACT else same > 0.99


@pytest.mark.parametrize("device", [True, False])
def test_uploads_of_one_build(device, want):
    scene = mixed().build(device=device)
    assert scene.built_on_device == device
    for _ in range(4):  # the tree of the build, a copy of the host's, the pinned image twice
        scene.upload()
        _check(scene, want)
        scene.release_device()
    # a change of the scene drops what was kept
    scene.add(zt.sphere((0, 0, 9), 0.5, 0))
    scene.build(device=device)
    changed = O.OracleScene.from_scene(scene).render(OPTS.width, OPTS.height, OPTS.spp, OPTS.max_depth, seed=OPTS.seed)
    _check(scene, changed)


@pytest.mark.parametrize("n", [1, 2, 5, 257])
def test_small_scenes(n):
    scene = mixed(n, seed=n).build(device=n % 2 == 1)
    want = O.OracleScene.from_scene(scene).render(OPTS.width, OPTS.height, OPTS.spp, OPTS.max_depth, seed=OPTS.seed)
    _check(scene, want)
    scene.release_device()
    _check(scene, want)


def test_rebuilt_without_an_upload(want):
    scene = mixed()
    for _ in range(3):
        scene.build(device=True)
    _check(scene, want)


def test_a_leaf_too_large_for_the_float_records(want):
    scene = mixed().build()
    nodes, idx = scene.bvh()
    # the first interior node whose subtree holds 16 or more shapes becomes a leaf of them
    size = nodes["count"].astype(np.int64)
    for i in np.flatnonzero(nodes["count"] == 0)[::-1]:
        size[i] = size[nodes["first"][i]] + size[nodes["first"][i] + 1]
    big = np.flatnonzero((nodes["count"] == 0) & (size >= 16) & (size <= 40))[-1]
    end = big
    while nodes["count"][end] == 0:
        end = nodes["first"][end]
    sub = [big]  # the subtree's nodes: children follow their parent
    for i in sub:
        if nodes["count"][i] == 0:
            sub += [nodes["first"][i], nodes["first"][i] + 1]
    gone = np.zeros(len(nodes), bool)
    gone[sub[1:]] = True
    new = np.cumsum(~gone) - 1
    out = nodes.copy()
    inner = (nodes["count"] == 0) & ~gone
    inner[big] = False
    out["first"][inner] = new[nodes["first"][inner]]
    out["first"][big], out["count"][big] = nodes["first"][end], size[big]
    scene.build_with_bvh(out[~gone], idx)
    fast = zt.render(scene, OPTS, zt.GpuConfig(precision=zt.PRECISION_FAST)).pixels
    exact = zt.render(scene, OPTS, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels
    assert fast.tobytes() == exact.tobytes()
    assert (exact == want).all(axis=1).mean() > 0.99


def test_nan_vertex():
    scene = mixed()
    scene.add(zt.triangle((0, 1, 0), (1, 1, 0), (float("nan"), 2, 0), 0))
    scene.build(device=True)
    a = zt.render(scene, OPTS).pixels
    assert a.tobytes() == zt.render(scene, OPTS, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels.tobytes()
