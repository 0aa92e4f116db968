"""The four-wide nodes of the LBVH, whose slots are opened by size: nearest hits equal to the oracle's at
the tree shapes where a node has two, three or four slots, for chains of ever smaller spheres (the deepest
trees, a leaf cluster beside every node) and for many spheres at one place (equal codes)."""
import numpy as np
import pytest

from ataraxia_gb300 import Renderer, scenes
from tests.helpers import bit_mismatches

pytestmark = pytest.mark.gpu


def _spheres(shape, n, rng):
    s = np.zeros(n, dtype=scenes.SPHERE_DTYPE)
    if shape == "box":
        c, r = rng.uniform(-10, 10, (n, 3)), rng.uniform(0.2, 1.0, n)
    elif shape == "chain":   # one more halving per sphere: a step of the tree each, as far as the codes reach
        at = 20.0 * 0.5 ** (np.arange(n) % 24)
        c, r = np.stack([at, -0.5 * at, 0.25 * at], axis=1), 0.1 * at
    else:   # one place, a few others
        c, r = np.zeros((n, 3)), rng.uniform(0.5, 1.0, n)
        c[::7] = rng.uniform(-10, 10, (len(c[::7]), 3))
    s["center"], s["radius"] = c, r
    return s


@pytest.mark.parametrize("shape", ["box", "chain", "one place"])
@pytest.mark.parametrize("leaf", [1, 8, 32])
@pytest.mark.parametrize("n", [2, 3, 5, 9, 17, 33, 70, 2000])
def test_nearest_hits(po, shape, leaf, n):
    rng = np.random.default_rng(n * 37 + leaf)
    sph = _spheres(shape, n, rng)
    sc = scenes.config0()
    d = rng.normal(size=(2000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    to = sph["center"][rng.integers(0, n, 2000)] + rng.normal(size=(2000, 3)) * sph["radius"].max()
    o, d = (to - rng.uniform(0, 30, (2000, 1)) * d).astype(np.float32), d.astype(np.float32)
    with Renderer(bvh_threshold=1, bvh_leaf_size=leaf) as r:
        r.set_scene(sph, sc.materials, sc.lights)
        t, i = r.trace_nearest(o, d)
    rt, ri = po.trace(sph, o, d, po.EXACT)
    assert np.array_equal(i, ri)
    assert bit_mismatches(t, rt) == 0
