"""Calls that do without a buffer where the device has no room for it, with
the device's memory held by another allocator of the process: the upload of a
scene whose block fits but not what the device flattening reads beside it.
Each runs in a process of its own, since what the library's pool already
holds decides what fits."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

COMMON = """
import numpy as np, torch
import zigtrace_b200 as zt

def spheres(n, seed):
    rng = np.random.default_rng(seed)
    s = zt.Scene()
    s.background = zt.Background.sky((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    m = [s.add_material(zt.Material.lambertian(tuple(rng.random(3)))) for _ in range(4)]
    s.add_spheres(rng.uniform(-10, 10, (n, 3)), np.full(n, 0.05), np.asarray(m)[np.arange(n) % 4])
    s.camera = zt.CameraConfig(look_from=(0.0, 0.0, 25.0), look_at=(0.0, 0.0, 0.0), vfov=50.0)
    return s

def hold_all_but(left):
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - int(left), dtype=torch.uint8, device="cuda")

o = zt.Options(64, 48, 2, 6, seed=1)
"""

UPLOAD = COMMON + """
device = {device}
small = spheres(500, 0).build(device=device)   # kernels and their local memory are loaded
zt.render(small, o)
n = 2_200_000 if device else 500_000           # of this size the build leaves nothing but the tree in the pool
scene = spheres(n, 1).build(device=device)
assert scene.built_on_device == device
block = scene.staging_bytes()
beside = 196 * n                               # shapes, permutation and nodes
held = hold_all_but(block + beside // 2 if not device else block - beside // 2)
img = zt.render(scene, o).pixels
del held
torch.cuda.empty_cache()
assert img.tobytes() == zt.render(spheres(n, 1).build(device=device), o).pixels.tobytes()
"""


def run(program):
    p = subprocess.run([sys.executable, "-c", program], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


@pytest.mark.parametrize("device", [False, True])
def test_upload_with_room_for_the_block_only(device):
    """device=True: the tree that the device build left makes room for it."""
    run(UPLOAD.format(device=device))


BUILD = COMMON + """
small = spheres(500, 0).build(device=True)
small.upload()
n = 2_500_000
scene = spheres(n, 1)
free = torch.cuda.mem_get_info()[0]
scene.build(device=True)
taken = free - torch.cuda.mem_get_info()[0]
assert scene.built_on_device
assert taken <= 196 * n + (64 << 20), taken    # shapes, permutation and nodes, until the upload
"""


def test_a_large_device_build_gives_its_scratch_back():
    run(BUILD)


GRADIENTS = COMMON + """
def many_materials(n):
    s = spheres(60, 3)
    rng = np.random.default_rng(5)
    m = np.concatenate([s.materials, np.tile(s.materials[:1], n)])
    m["color"][4:] = rng.random((n, 3))
    t = zt.Scene()
    t.background, t.camera = s.background, s.camera
    t.add_materials(m)
    t.add_shapes(s.shapes)
    return t

g = np.ones((o.width * o.height, 3))
few = many_materials(8).build()
zt.forward(few, o)
zt.backward(few, o, g)
scene = many_materials(200_000).build()
zt.forward(scene, o)
held = hold_all_but(24 << 20)                  # a slice of gradients is 4.8 MB, all slices 64 MB
got = zt.backward(scene, o, g)
del held
torch.cuda.empty_cache()
want = zt.backward(scene, o, g)
assert np.abs(want).max() > 1
np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-11 * np.abs(want).max())
"""


def test_backward_with_room_for_few_gradient_slices():
    """Sums of at most 64 x 48 x 2 x 6 terms in another order."""
    run(GRADIENTS)
