"""The checked float walk on the GPU: the default precision of scenes with
at least 64 bounded primitives, bit-identical to the oracle or to the f64
walk (the wavefront tracer keeps it), also where every hit is a tie, where
the tree's boxes do not hold their primitives, and where rays come from
beyond the float test's range."""
import numpy as np
import pytest

import kat_scenes as K
import oracle as O
import zigtrace_b200 as zt
from zigtrace_b200 import scenes

pytestmark = pytest.mark.gpu

MODES = [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN]


def _icosphere(scene, center, radius, material):
    verts, faces = scenes.icosphere(2)
    v = np.asarray(verts) * radius + np.asarray(center, float)
    f = np.asarray(faces)
    scene.add_triangles(v[f[:, 0]], v[f[:, 1]], v[f[:, 2]], material)
    return scene


def doubled():
    """Every triangle of an icosphere and of the floor twice, with another
    material the second time: each hit is a tie."""
    s = scenes.cornell()
    glow = s.add_material(zt.Material.emissive((0.2, 0.4, 0.1)))
    _icosphere(s, (250, 250, 250), 90.0, 2)
    _icosphere(s, (250, 250, 250), 90.0, glow)
    s.add_quad((0, 0, 0), (555, 0, 0), (0, 0, 555), 0)
    return s


def far_plane():
    """Grazing bounces off a plane reach hits beyond 1e30 only with luck;
    a camera far along it makes distant origins common."""
    s = scenes.random_spheres(3, grid=12)
    s.camera = zt.CameraConfig(look_from=(9e6, 2, 3), look_at=(0, 0, 0), vfov=0.001, aperture=0.0)
    return s


SCENES = {"fuzz2": lambda: _icosphere(K.fuzz_scene(2), (1.5, 0.6, -3.5), 0.5, 0),
          "fuzz6": lambda: _icosphere(K.fuzz_scene(6), (0.5, 0.4, -2.5), 0.4, 1),
          "cornell": lambda: _icosphere(scenes.cornell(), (400, 330, 200), 60.0, 2),
          "spheres": lambda: scenes.random_spheres(5), "doubled": doubled, "far_plane": far_plane,
          "terrain": lambda: scenes.triangle_heavy(2, nx=60, nz=30, n_ico=4, ico_subdiv=2, n_lights=9)}


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("name", SCENES)
def test_bit_identical_to_the_oracle(name, mode):
    scene = SCENES[name]().build()
    assert scene.counts()["bounded"] >= 64
    o = zt.Options(61, 37, 6, 12, seed=4)
    img = zt.render(scene, o, zt.GpuConfig(mode)).pixels
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert img.tobytes() == want.tobytes()


@pytest.mark.parametrize("name", ["spheres", "doubled"])
def test_batch_bit_identical(name):
    scene = SCENES[name]().build()
    o = zt.Options(45, 31, 4, 10, seed=2)
    img = zt.render_batch([scene, scene], [o, o])
    want = O.OracleScene.from_scene(scene).render(o.width, o.height, o.spp, o.max_depth, seed=o.seed)
    assert img[0].pixels.tobytes() == want.tobytes() and img[1].pixels.tobytes() == want.tobytes()


@pytest.mark.parametrize("mode", MODES)
def test_imported_tree_whose_boxes_cut_their_primitives(mode):
    """Leaf boxes shrunk to a third: the f64 walk misses most primitives, and
    so must this one."""
    scene = SCENES["cornell"]()
    scene.build()
    nodes, idx = scene.bvh()
    leaf = nodes["count"] > 0
    mid = 0.5 * (nodes["bmin"] + nodes["bmax"])
    for k in ("bmin", "bmax"):
        nodes[k][leaf] = mid[leaf] + (nodes[k][leaf] - mid[leaf]) / 3
    scene.build_with_bvh(nodes, idx)
    o = zt.Options(48, 40, 4, 8, seed=1)
    img = zt.render(scene, o, zt.GpuConfig(mode)).pixels
    assert img.tobytes() == zt.render(scene, o, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels.tobytes()


def test_nan_vertex_renders_as_the_f64_walk():
    scene = SCENES["spheres"]()
    scene.add(zt.triangle((0, 1, 0), (1, 1, 0), (float("nan"), 2, 0), 0))
    scene.build()
    o = zt.Options(40, 30, 2, 6, seed=1)
    assert zt.render(scene, o).pixels.tobytes() == zt.render(scene, o, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels.tobytes()
