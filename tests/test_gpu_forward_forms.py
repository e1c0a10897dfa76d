"""The differentiable forward on scenes whose paths are short (nested: a lane
waits for its warp's longest path) and long (path regeneration), on images
whose tiles are split and whole: at the scene's own colours the oracle's
image, and the samples it keeps give the backward the gradients that it finds
without them."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu

SCENES = {"open": lambda: scenes.random_spheres(4, grid=8), "closed": scenes.cornell,
          "mesh": lambda: scenes.triangle_heavy(1, nx=60, nz=30, n_ico=3, ico_subdiv=2, n_lights=5)}


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("w,h", [(1, 1), (9, 5), (61, 33), (190, 107), (333, 217)])
def test_image_and_gradients(name, w, h):
    scene = SCENES[name]().build()
    o = zt.Options(w, h, 3, 7, seed=w)
    img = zt.forward(scene, o).pixels
    want = O.OracleScene.from_scene(scene).render(w, h, 3, 7, seed=w)
    assert img.tobytes() == want.tobytes()
    g = np.random.default_rng(w).normal(size=(w * h, 3))
    kept = zt.backward(scene, o, g)
    scene.set_primal_cache_limit(0)
    zt.forward(scene, o)
    traced = zt.backward(scene, o, g)
    # the same terms in another order: at most w h 3 7 of them a parameter
    scale = np.abs(traced).max() + 1e-300
    np.testing.assert_allclose(kept, traced, rtol=0, atol=scale * w * h * 21 * 2.0 ** -52 * 4)
