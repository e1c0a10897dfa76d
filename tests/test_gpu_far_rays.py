"""Rays from beyond what the float box test takes (zt_fast.cuh,
kFastMaxOrigin): camera rays leave a scene, meet a mirror plane far below it
and come back through it from there.  Their pixels must take the f64 walk, in
every kernel form and at both precisions."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu


def far_mirror(distance, floor=zt.Material.metal((0.9, 0.8, 0.7), 0.0)):
    """Triangles and spheres above a camera that looks straight down at a
    plane `distance` below; a view just wide enough for the reflected rays to
    spread over the scene."""
    rng = np.random.default_rng(11)
    s = zt.Scene()
    s.background = zt.Background.sky((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    mats = [s.add_material(m) for m in (zt.Material.lambertian((0.2, 0.6, 0.3)), zt.Material.lambertian((0.7, 0.3, 0.2)),
                                        zt.Material.dielectric(1.5), zt.Material.emissive((3.0, 2.0, 1.0)))]
    for k in range(120):
        c = np.array([rng.uniform(-9, 9), rng.uniform(40, 60), rng.uniform(-9, 9)])
        if k % 3:
            a, b = rng.uniform(0.5, 2.5, 2)
            s.add(zt.triangle(c, c + [a, 0, 0], c + [0, rng.uniform(-0.5, 0.5), b], mats[k % 4]))
        else:
            s.add(zt.sphere(c, rng.uniform(0.3, 1.2), mats[k % 4]))
    s.add(zt.plane((0.0, -distance, 0.0), (0.0, 1.0, 0.0), s.add_material(floor)))
    s.camera = zt.CameraConfig(look_from=(0.0, 0.0, 0.0), look_at=(0.0, -1.0, 0.0), up=(0.0, 0.0, 1.0),
                               vfov=float(np.degrees(10.0 / distance)))
    return s


def oracle_image(scene, o):
    return O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)


@pytest.mark.parametrize("distance", [3e8, 4e9, 1e12, 3e19, 1e31, 1e39])
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
def test_bit_identical_to_the_oracle(distance, mode):
    scene = far_mirror(distance).build()
    o = zt.Options(45, 29, 4, 8, seed=3)
    want = oracle_image(scene, o)
    assert len(np.unique(want, axis=0)) > o.width * o.height // 10  # the scene is seen, not the sky alone
    assert zt.render(scene, o, zt.GpuConfig(mode)).pixels.tobytes() == want.tobytes()


@pytest.mark.parametrize("distance", [1e12, 3e19, 1e39])
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
def test_the_fast_precision_takes_the_f64_walk_there(distance, mode):
    """Every path of this view goes by way of the mirror."""
    scene = far_mirror(distance).build()
    o = zt.Options(45, 29, 4, 8, seed=3)
    img = zt.render(scene, o, zt.GpuConfig(mode, precision=zt.PRECISION_FAST)).pixels
    assert img.tobytes() == oracle_image(scene, o).tobytes()


@pytest.mark.parametrize("precision", [zt.PRECISION_EXACT, zt.PRECISION_FAST])
def test_batch_and_shadow_rays(precision):
    """A diffuse plane far below: light samples and bounces start there."""
    scene = far_mirror(3e19, zt.Material.lambertian((0.6, 0.6, 0.6))).build()
    mirror = far_mirror(1e31).build()
    o = zt.Options(37, 22, 4, 6, seed=9)
    imgs = zt.render_batch([scene, mirror], [o, o], zt.GpuConfig(precision=precision))
    for s, img in zip((scene, mirror), imgs):
        assert img.pixels.tobytes() == oracle_image(s, o).tobytes()
