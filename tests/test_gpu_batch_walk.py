"""The walk of a batch at the default precision: the f64 walk where most of its
work is on scenes too small for the checked float walk to pay (the Cornell
box), the checked walk elsewhere; every image the oracle's."""
import pytest

import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes,fields", [(3, 0), (5, 1), (1, 3), (0, 2)])
@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
def test_mixed_batches_bit_identical(boxes, fields, mode):
    scs = [scenes.cornell() for _ in range(boxes)] + [scenes.random_spheres(k, grid=10) for k in range(fields)]
    opts = [zt.Options(33 + k, 21, 4, 8, seed=k) for k in range(len(scs))]
    for s in scs:
        s.build()
    for s, o, img in zip(scs, opts, zt.render_batch(scs, opts, zt.GpuConfig(mode))):
        want = O.OracleScene.from_scene(s).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
        assert img.pixels.tobytes() == want.tobytes()
