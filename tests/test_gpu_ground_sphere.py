"""The default precision over a ground made of a large sphere: where its box
touches the sphere the checked walk's hits used to be in doubt.  Bit-identical
to the oracle, near the pole and away from it."""
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def ground_sphere(radius):
    s = scenes.random_spheres(6, grid=12)
    shapes = s.shapes.copy()
    g = shapes["kind"] == zt.PLANE
    assert g.sum() == 1
    shapes["kind"][g] = zt.SPHERE
    shapes["p"][g] = 0.0
    shapes["p"][g, 1], shapes["p"][g, 3] = -radius, radius
    t = zt.Scene()
    t.background, t.camera = s.background, s.camera
    t.add_materials(s.materials)
    t.add_shapes(shapes)
    return t


@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
@pytest.mark.parametrize("radius", [1000.0, 5000.0, 1e5, 4e6])
def test_bit_identical_to_the_oracle(radius, mode):
    scene = ground_sphere(radius).build()
    o = zt.Options(121, 67, 16, 20, seed=2)
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert zt.render(scene, o, zt.GpuConfig(mode)).pixels.tobytes() == want.tobytes()


def test_straight_down_on_the_pole():
    scene = ground_sphere(1000.0)
    scene.camera = zt.CameraConfig(look_from=(0.01, 40.0, 0.02), look_at=(0.01, 0.0, 0.02), up=(0.0, 0.0, 1.0),
                                   vfov=0.02)
    scene.build()
    o = zt.Options(64, 64, 8, 10, seed=5)
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert zt.render(scene, o).pixels.tobytes() == want.tobytes()
