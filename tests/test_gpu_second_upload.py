"""The second upload of a build keeps a page-locked image of the scene, so that
later ones are one copy.  Making it may not cost more than building the scene
again on the device would; the images of all uploads are the same."""
import time

import numpy as np
import pytest

import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def test_second_upload_costs_less_than_a_build():
    import torch
    build, second, images = [], [], set()
    o = zt.Options(96, 54, 2, 8, seed=1)
    for rep in range(4):
        scene = scenes.triangle_heavy(0)
        scene.shapes
        t = time.perf_counter()
        scene.build(device=True)
        build.append(time.perf_counter() - t)
        for k in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            scene.upload()
            torch.cuda.synchronize()
            if k == 1:
                second.append(time.perf_counter() - t)
            images.add(zt.render(scene, o).pixels.tobytes())
            scene.release_device()
    assert len(images) == 1
    assert np.min(second) <= np.min(build[1:]), (second, build)


@pytest.mark.parametrize("n", [200, 12_000, 16_000, 90_000])
def test_images_on_both_sides_of_the_huge_page_size(n):
    """276 bytes a sphere: below and from 4 MB up."""
    rng = np.random.default_rng(n)
    s = zt.Scene()
    s.background = zt.Background.sky((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    m = s.add_material(zt.Material.lambertian((0.5, 0.4, 0.3)))
    s.add_spheres(rng.uniform(-10, 10, (n, 3)), np.full(n, 0.1), m)
    s.camera = zt.CameraConfig(look_from=(0.0, 0.0, 25.0), look_at=(0.0, 0.0, 0.0), vfov=50.0)
    s.build()
    o = zt.Options(64, 48, 2, 6, seed=1)
    images = set()
    for _ in range(4):
        images.add(zt.render(s, o).pixels.tobytes())
        s.release_device()
    assert len(images) == 1
