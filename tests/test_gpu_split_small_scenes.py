"""Images of a scene too small for the float walk, rendered by the nested
kernel on both sides of each size at which its 8x4 tiles are split further
(3/8 of the resident warps): every pixel equals the oracle's."""
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(80, 40), (104, 68), (120, 60), (145, 99), (160, 92), (232, 121), (233, 128), (256, 144)])
def test_every_pixel(w, h):
    scene = scenes.cornell().build()
    o = zt.Options(w, h, 2, 8, seed=h)
    img = zt.render(scene, o, zt.GpuConfig(zt.MODE_MEGAKERNEL)).pixels
    assert img.tobytes() == O.OracleScene.from_scene(scene).render(w, h, 2, 8, seed=h).tobytes()
