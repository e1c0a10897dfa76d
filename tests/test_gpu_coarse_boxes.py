"""Scenes whose reach, or whose camera's distance, is so large beside their
objects that the float boxes' margins cover several of them: the default
precision gives the oracle's image and does not visit every object with every
ray (ZT_PRECISION_FAST, which keeps the float boxes, does)."""
import dataclasses

import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt
from test_gpu_ground_sphere import ground_sphere
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def on_a_square(half):
    s = scenes.random_spheres(0, grid=16)
    t = zt.Scene()
    t.background, t.camera = s.background, s.camera
    t.add_materials(s.materials)
    t.add_shapes(s.shapes[s.shapes["kind"] != zt.PLANE])
    t.add_quad((-half, -0.001, -half), (0, 0, 2 * half), (2 * half, 0, 0), 0)
    return t


def seen_from(distance):
    s = scenes.random_spheres(0, grid=16)
    at, to = np.array(s.camera.look_from), np.array(s.camera.look_at)
    d = (at - to) / np.linalg.norm(at - to)
    s.camera = dataclasses.replace(s.camera, look_from=tuple(to + d * distance), vfov=float(np.degrees(8 / distance)),
                                   aperture=0.0)
    return s


SCENES = {"square_1e4": lambda: on_a_square(1e4), "square_1e5": lambda: on_a_square(1e5),
          "square_4e5": lambda: on_a_square(4e5), "square_9e6": lambda: on_a_square(9e6),
          "sphere_4e6": lambda: ground_sphere(4e6), "from_1e5": lambda: seen_from(1e5),
          "from_9e6": lambda: seen_from(9e6)}


@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
def test_bit_identical_to_the_oracle(name, mode):
    scene = SCENES[name]().build()
    o = zt.Options(61, 37, 4, 12, seed=4)
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert zt.render(scene, o, zt.GpuConfig(mode)).pixels.tobytes() == want.tobytes()


@pytest.mark.parametrize("name", ["square_9e6", "sphere_4e6"])
def test_the_default_precision_avoids_coarse_boxes(name):
    """The float walk takes 66 and 42 ms at 1280x720x16 where the f64 walk
    takes 5.7 and 5.4: more than seven times as long."""
    import torch
    scene = SCENES[name]().build()
    scene.upload()
    o = zt.Options(640, 360, 8, 20, seed=1)
    out = torch.empty(3 * o.width * o.height, dtype=torch.float64, device="cuda")
    best = {}
    for precision in (zt.PRECISION_EXACT, zt.PRECISION_FAST) * 4:
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        zt.render_device(scene, o, out.data_ptr(), 0, zt.GpuConfig(precision=precision))
        b.record()
        torch.cuda.synchronize()
        best[precision] = min(best.get(precision, np.inf), a.elapsed_time(b))
    assert best[zt.PRECISION_EXACT] <= 0.5 * best[zt.PRECISION_FAST], best
