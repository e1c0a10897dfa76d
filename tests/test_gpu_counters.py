"""A bounce limit beyond 32 bits, which the float-walk kernels' counters do
not hold: such a render takes the f64 walk and equals the one whose limit no
path reaches."""
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [2 ** 32 - 1, 2 ** 32, 2 ** 32 + 3, 2 ** 40])
@pytest.mark.parametrize("precision", [zt.PRECISION_EXACT, zt.PRECISION_FAST])
def test_bounce_limits_beyond_32_bits(depth, precision):
    scene = scenes.random_spheres(1, grid=10).build()
    img = zt.render(scene, zt.Options(40, 24, 3, depth, seed=2), zt.GpuConfig(precision=precision)).pixels
    want = O.OracleScene.from_scene(scene).render(40, 24, 3, 1000, seed=2)
    assert img.tobytes() == want.tobytes()
