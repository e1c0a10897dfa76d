"""The differentiable pair at its edges: images that are not whole tiles, one
sample, zero adjoints, more parameters than there are slices' bytes for, row
bands -- the cached backward, the uncached one and the bands' shares agree,
and the adjoint matches central differences along a random direction."""
import numpy as np
import pytest

import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def _close(a, b):
    """Equal up to the order of additions: 1e-12 of the largest entry."""
    assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (1, 1, 7), (7, 5, 3), (33, 9, 1), (9, 41, 4), (64, 32, 2)])
def test_cached_uncached_and_bands_agree(w, h, spp):
    scene, colors = scenes.cornell_diff(2)
    scene.build()
    o = zt.Options(w, h, spp, 12, seed=5)
    rng = np.random.default_rng(w * h)
    g = rng.normal(size=(w * h, 3))
    g[rng.random(w * h) < 0.3] = 0.0
    if w * h == 1:
        g[:] = 1.0
    img = zt.forward(scene, o, colors).pixels
    cached = zt.backward(scene, o, g, colors)
    scene.set_primal_cache_limit(0)
    assert zt.forward(scene, o, colors).pixels.tobytes() == img.tobytes()
    _close(zt.backward(scene, o, g, colors), cached)
    cut = (h + 1) // 2
    bands = [(0, cut)] + ([(cut, h)] if cut < h else [])
    _close(sum(zt.backward_rows(scene, o, a, b, g[a * w:b * w], colors) for a, b in bands), cached)
    step = rng.normal(size=colors.shape) * colors * 1e-4
    diff = (zt.forward(scene, o, colors + step).pixels - zt.forward(scene, o, colors - step).pixels) / 2
    # third-order remainder of a relative step of 1e-4, and the images' rounding
    scale = np.abs(g * img).sum()
    assert abs((diff * g).sum() - (cached * step).sum()) <= 1e-7 * scale + 1e-13 * scale


@pytest.mark.parametrize("materials", [2, 700, 200_000])
def test_any_number_of_parameters(materials):
    rng = np.random.default_rng(materials)
    s = zt.Scene()
    s.background = zt.Background.solid((0.3, 0.4, 0.5))
    mats = np.zeros(materials, dtype=s.materials.dtype)
    mats["kind"] = zt.LAMBERTIAN
    mats["color"] = rng.uniform(0.2, 0.9, (materials, 3))
    mats["kind"][-1], mats["color"][-1] = zt.EMISSIVE, (4.0, 5.0, 6.0)
    s.add_materials(mats)
    c = rng.uniform(-2, 2, (200, 3))
    s.add_triangles(c, c + rng.uniform(-1, 1, c.shape), c + rng.uniform(-1, 1, c.shape),
                    rng.integers(0, materials - 1, 200))
    s.add_quad((-1, 3, -1), (2, 0, 0), (0, 0, 2), materials - 1)
    s.camera = zt.CameraConfig(look_from=(0, 0, 7))
    s.build()
    o = zt.Options(30, 21, 4, 6, seed=1)
    colors = s.materials["color"].copy()
    img = zt.forward(s, o, colors).pixels
    g = rng.normal(size=img.shape)
    grad = zt.backward(s, o, g, colors)
    used = np.zeros(materials, bool)
    used[s.shapes["material"]] = True
    assert (grad[~used] == 0).all() and (grad[used] != 0).any()
    s.set_primal_cache_limit(0)
    _close(zt.backward(s, o, g, colors), grad)
