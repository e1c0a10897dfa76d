"""Images of few pixels, whose 8x4 tiles are rendered in up to 16 parts by a
warp each: every pixel is rendered once and equals the oracle's, whole images
and row bands, nested and regenerating, and the differentiable forward."""
import pytest

import kat_scenes as K
import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu

SCENES = {"fuzz": lambda: K.fuzz_scene(4), "spheres": lambda: scenes.random_spheres(2, grid=10)}
# sixteenths down to whole tiles of the regenerating and of the nested kernels
SIZES = [(1, 1), (2, 3), (8, 4), (9, 5), (65, 33), (130, 61), (250, 77), (333, 217)]


@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
@pytest.mark.parametrize("name", SCENES)
@pytest.mark.parametrize("w,h", SIZES)
def test_every_pixel(w, h, name, mode):
    scene = SCENES[name]().build()
    o = zt.Options(w, h, 2, 6, seed=w)
    img = zt.render(scene, o, zt.GpuConfig(mode)).pixels
    want = O.OracleScene.from_scene(scene).render(w, h, 2, 6, seed=w)
    assert img.tobytes() == want.tobytes()


@pytest.mark.parametrize("w,h,y0,y1", [(37, 20, 3, 4), (37, 20, 7, 20), (200, 90, 41, 90), (400, 300, 1, 300)])
def test_bands(w, h, y0, y1):
    import torch
    scene = SCENES["spheres"]().build()
    scene.upload()
    o = zt.Options(w, h, 2, 6, seed=1)
    want = O.OracleScene.from_scene(scene).render(w, h, 2, 6, seed=1).reshape(h, w, 3)[y0:y1]
    out = torch.zeros((y1 - y0, w, 3), dtype=torch.float64, device="cuda")
    zt.render_rows_device(scene, o, y0, y1, out.data_ptr())
    assert out.cpu().numpy().tobytes() == want.tobytes()
    assert zt.forward_rows(scene, o, y0, y1).tobytes() == want.tobytes()
