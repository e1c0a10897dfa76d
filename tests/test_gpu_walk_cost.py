"""The default precision renders a pixel again with the f64 walk where a hit of
its float walk is in doubt.  That must stay the exception on scenes whose
geometry coincides or touches its boxes: the default precision of such a scene
may take half as long again as ZT_PRECISION_FAST (the same walk without the
check), which a pixel in thirty rendered twice by one lane of its warp
exceeds."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt
from test_gpu_ground_sphere import ground_sphere
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def terrain_with_copies(every):
    """Each `every`-th triangle a second time, with another material."""
    s = scenes.triangle_heavy(0, nx=200, nz=100)
    red = s.add_material(zt.Material.lambertian((0.7, 0.2, 0.1)))
    again = s.shapes[::every].copy()
    again["material"] = red
    s.add_shapes(again)
    return s


SCENES = {"ground_sphere": lambda: ground_sphere(1000.0), "each_twice": lambda: terrain_with_copies(1),
          "some_twice": lambda: terrain_with_copies(50)}


@pytest.mark.parametrize("name", SCENES)
def test_few_pixels_are_rendered_twice(name):
    import torch
    scene = SCENES[name]().build()
    scene.upload()
    o = zt.Options(640, 360, 16, 12, seed=1)
    out = torch.empty(3 * o.width * o.height, dtype=torch.float64, device="cuda")
    best = {}
    for precision in (zt.PRECISION_EXACT, zt.PRECISION_FAST) * 6:
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        zt.render_device(scene, o, out.data_ptr(), 0, zt.GpuConfig(precision=precision))
        b.record()
        torch.cuda.synchronize()
        best[precision] = min(best.get(precision, np.inf), a.elapsed_time(b))
    assert best[zt.PRECISION_EXACT] <= 1.5 * best[zt.PRECISION_FAST], best


@pytest.mark.parametrize("every", [1, 50])
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
def test_coincident_triangles_bit_identical_to_the_oracle(every, mode):
    """The first of two coincident triangles keeps the hit."""
    scene = terrain_with_copies(every).build()
    o = zt.Options(61, 37, 4, 8, seed=4)
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert zt.render(scene, o, zt.GpuConfig(mode)).pixels.tobytes() == want.tobytes()
