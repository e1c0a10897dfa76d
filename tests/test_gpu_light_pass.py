"""Scenes with many lights on the GPU, bit-identical to the oracle: touching
and overlapping quads, slivers, spheres and lights seen edge-on, all of them
reached by bounces, so that the emission pdf's light loop decides."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


def many_lights(n):
    rng = np.random.default_rng(n)
    s = zt.Scene()
    s.background = zt.Background.solid((0.0, 0.0, 0.0))
    floor = s.add_material(zt.Material.lambertian((0.7, 0.6, 0.5)))
    lamps = [s.add_material(zt.Material.emissive(rng.uniform(1, 8, 3))) for _ in range(4)]
    s.add(zt.plane((0, 0, 0), (0, 1, 0), floor))
    verts, faces = scenes.icosphere(1)
    v = verts + np.array([0, 1.0, 0])
    s.add_triangles(v[faces[:, 0]], v[faces[:, 1]], v[faces[:, 2]], floor)
    for k in range(n):
        x, z = rng.uniform(-4, 3, 2)
        lamp = lamps[k % 4]
        if k % 7 == 3:
            s.add(zt.sphere((x, 2.5, z), 0.3, lamp))
        elif k % 7 == 5:
            s.add(zt.triangle((x, 2.2, z), (x + 2, 2.2, z), (x + 1, 2.2, z + 1e-3), lamp))
        elif k % 7 == 6:  # standing
            s.add_quad((x, 0.2, z), (0, 2.0, 0), (0.5, 0, 0.5), lamp)
        else:  # facing down, two heights: many overlap
            s.add_quad((x, 3.0 + (k % 2) * 1e-7, z), (1.0, 0, 0), (0, 0, 1.0), lamp)
    s.camera = zt.CameraConfig(look_from=(0, 2, 7), look_at=(0, 1, 0), vfov=60)
    return s


@pytest.mark.parametrize("precision", [zt.PRECISION_EXACT, zt.PRECISION_FAST])
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
@pytest.mark.parametrize("n", [1, 40, 150])
def test_many_lights_bit_identical(n, mode, precision):
    scene = many_lights(n).build()
    o = zt.Options(57, 39, 8, 10, seed=3)
    img = zt.render(scene, o, zt.GpuConfig(mode, precision=precision)).pixels
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    same = (img == want).all(axis=1).mean()
    assert same == 1.0 if precision == zt.PRECISION_EXACT else same > 0.99
