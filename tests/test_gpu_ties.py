"""Exact ties between leaves in the checked walk (tie_first, zt_fast.cuh):
overlapping faces in common planes, whose vertices lie on a coarse grid so
that distances agree to the last bit, each with a material of its own.  The
primitive that the f64 walk tests first keeps the hit: bit-identical to the
oracle, from the host's and the device's trees, and from an imported tree
whose leaves are not in the tree's order, where no order can be shown."""
import numpy as np
import pytest

import oracle as O
import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu


def flush_faces(seed, n=160):
    """Squares and triangles on the planes x, y, z = 0 .. 4 of a small grid."""
    rng = np.random.default_rng(seed)
    s = zt.Scene()
    s.background = zt.Background.sky((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    mats = [s.add_material(zt.Material.lambertian(tuple(rng.uniform(0.1, 0.9, 3)))) for _ in range(24)]
    mats += [s.add_material(zt.Material.emissive(tuple(rng.uniform(0.5, 4.0, 3)))) for _ in range(4)]
    mats += [s.add_material(zt.Material.metal((0.8, 0.8, 0.8), 0.0))]
    for _ in range(n):
        ax = rng.integers(0, 3)
        c = rng.integers(0, 5, 3).astype(float)
        u, v = np.zeros(3), np.zeros(3)
        u[(ax + 1) % 3], v[(ax + 2) % 3] = rng.choice([1.0, 2.0, 4.0], 2)
        if rng.random() < 0.5:
            u, v = v, u
        m = mats[rng.integers(0, len(mats))]
        if rng.random() < 0.7:
            s.add_quad(tuple(c), tuple(u), tuple(v), m)
        else:
            s.add(zt.triangle(tuple(c), tuple(c + u), tuple(c + v), m))
    s.camera = zt.CameraConfig(look_from=(9.0, 7.0, 11.0), look_at=(2.0, 2.0, 2.0), vfov=45.0)
    return s


def flush_light():
    """A closed box with its light in the plane of its ceiling, and a mesh."""
    from zigtrace_b200 import scenes
    s = scenes.cornell()
    glow = s.add_material(zt.Material.emissive((9.0, 8.0, 7.0)))
    top = s.shapes["p"][s.shapes["kind"] == zt.TRIANGLE].reshape(-1, 3)[:, 1].max()
    s.add_quad((180.0, float(top), 180.0), (200.0, 0.0, 0.0), (0.0, 0.0, 200.0), glow)
    verts, faces = scenes.icosphere(2)
    v, f = np.asarray(verts) * 70.0 + (400.0, 330.0, 200.0), np.asarray(faces)
    s.add_triangles(v[f[:, 0]], v[f[:, 1]], v[f[:, 2]], 0)
    return s


def mirrored(scene):
    """The same tree with the children of every node exchanged: its leaves lie
    right to left."""
    scene.build()
    nodes, idx = scene.bvh()
    inner = np.flatnonzero(nodes["count"] == 0)
    out = nodes.copy()
    for i in inner:
        a = nodes["first"][i]
        out[a], out[a + 1] = nodes[a + 1], nodes[a]
    return scene.build_with_bvh(out, idx)


SCENES = {**{f"faces{s}": (lambda s=s: flush_faces(s)) for s in range(6)}, "light": flush_light}
O_ = zt.Options(64, 41, 6, 8, seed=7)


def want(scene):
    return O.OracleScene.from_scene(scene).render(O_.width, O_.height, O_.spp, O_.max_depth, seed=O_.seed)


@pytest.mark.parametrize("mode", [zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN])
@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("name", SCENES)
def test_bit_identical_to_the_oracle(name, device, mode):
    scene = SCENES[name]().build(device=device)
    assert scene.counts()["bounded"] >= 64
    img = zt.render(scene, O_, zt.GpuConfig(mode)).pixels
    assert img.tobytes() == want(scene).tobytes()


@pytest.mark.parametrize("name", ["faces1", "light"])
def test_leaves_out_of_the_trees_order(name):
    scene = mirrored(SCENES[name]())
    f64 = zt.render(scene, O_, zt.GpuConfig(zt.MODE_WAVEFRONT)).pixels
    for _ in range(3):  # from the device flattening twice, and the pinned image
        for mode in (zt.MODE_MEGAKERNEL, zt.MODE_MEGAKERNEL_REGEN):
            assert zt.render(scene, O_, zt.GpuConfig(mode)).pixels.tobytes() == f64.tobytes()
        scene.release_device()


def test_batch():
    scenes_ = [SCENES["faces2"]().build(), SCENES["light"]().build()]
    for s, img in zip(scenes_, zt.render_batch(scenes_, [O_, O_])):
        assert img.pixels.tobytes() == want(s).tobytes()


def test_a_light_flush_with_the_ceiling_costs_no_second_rendering():
    import torch
    scene = flush_light().build()
    scene.upload()
    o = zt.Options(400, 400, 16, 12, seed=1)
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
