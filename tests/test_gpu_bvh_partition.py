"""The device build's partition where its element chains are long, and its
nodes of one and two primitives: node for node and index for index the host
build's tree."""
import numpy as np
import pytest

import zigtrace_b200 as zt

pytestmark = pytest.mark.gpu


def _spheres(x, y=None, z=None, r=None):
    s = zt.Scene()
    m = s.add_material(zt.Material.lambertian((0.5, 0.5, 0.5)))
    n = len(x)
    c = np.stack([x, np.zeros(n) if y is None else y, np.zeros(n) if z is None else z], axis=1)
    s.add_spheres(c, np.full(n, 0.01) if r is None else r, m)
    return s


def _one_right_in_front(n):
    """The first element alone goes right: the displaced element's chain
    passes every other position."""
    x = np.linspace(0.0, 1.0, n)
    x[0] = 40.0
    return _spheres(x)


def _few_right(n):
    x = np.random.default_rng(n).random(n)
    x[::997] += 30.0
    return _spheres(x)


def _pairs(n):
    """Pairs that touch, coincide, share a coordinate or lie apart: two
    primitives split or stay a leaf."""
    rng = np.random.default_rng(n)
    c = rng.uniform(-50, 50, (n, 3))
    d = rng.choice([0.0, 0.005, 0.02, 0.5], (n, 3)) * rng.choice([-1, 1], (n, 3))
    p = np.stack([c, c + d], axis=1).reshape(-1, 3)[rng.permutation(2 * n)]
    return _spheres(p[:, 0], p[:, 1], p[:, 2], rng.choice([0.01, 0.2], 2 * n))


SCENES = {"front_33": lambda: _one_right_in_front(33), "front_70": lambda: _one_right_in_front(70),
          "front_5000": lambda: _one_right_in_front(5000), "front_120001": lambda: _one_right_in_front(120001),
          "few_40000": lambda: _few_right(40000), "pairs_1": lambda: _pairs(1), "pairs_20": lambda: _pairs(20),
          "pairs_30000": lambda: _pairs(30000),
          "descending": lambda: _spheres(np.linspace(1, 0, 9000)),
          "alternating": lambda: _spheres(np.tile([0.0, 1.0], 4500) + np.arange(9000) * 1e-6)}


@pytest.mark.parametrize("name", SCENES)
def test_same_tree(name):
    dev, host = SCENES[name]().build(device=True), SCENES[name]().build()
    n1, i1 = dev.bvh()
    n2, i2 = host.bvh()
    assert dev.built_on_device
    assert (i1 == i2).all()
    for k in ("first", "count", "bmin", "bmax"):
        assert (n1[k] == n2[k]).all(), k
