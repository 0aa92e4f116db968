"""Primary hits by warp cones (csrc/wavefront.cu k_primary, k_tile_masks, k_tile_lists) at images that end
inside a tile of 8 x 4 pixels and waves that do, with a moved camera (caps or the cone's walk) and with a camera
that stayed (tile masks or lists): frames equal the oracle bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


# a few tiles and a rest in both directions, whole tiles, narrower than a tile, one pixel across, one wide row
# of tiles; up to 32 mask words, and tables past the staged caps; leaf clusters up to and past 16 spheres; more
# and fewer than two pixels a sphere; one wave and many small ones that start and end inside tiles
@pytest.mark.parametrize("wave", [0, 700])
@pytest.mark.parametrize("res", [(95, 31), (32, 24), (7, 30), (1, 5), (1281, 3)])
@pytest.mark.parametrize("n,threshold,leaf", [(40, 1 << 30, 0), (1024, 1 << 30, 0), (1100, 1 << 30, 0), (700, 1, 0),
                                              (700, 1, 24), (5, 1, 1)])
def test_tiles_bit_exact(po, res, n, threshold, leaf, wave):
    st = scenes.Stream(17, f"rows{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(0.0, 0.5, n), st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.0 * half))
    sc = scenes.SyntheticScene("rows", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, 3, 1.5 * half), pos, d,
                               width=res[0], height=res[1], max_bounces=2, spp=1)
    view = po.view_for(sc)
    with Renderer(bvh_threshold=threshold, bvh_leaf_size=leaf, wave_paths=wave) as r:
        r.on_resize(*res)
        r.set_tuning(path_kernel=1, bvh_leaf_size=leaf, wave_paths=wave)
        r.set_scene(s, sc.materials, sc.lights)
        r.set_settings(Settings(maxBounces=2))
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        for k in (1, 2, 1):   # the camera's tables are built on its second render
            r.render_frames(k)
        got = r.get_accumulation().reshape(-1, 4)
    want, _, _ = oracle_render(sc, 4)
    assert bit_mismatches(got, want) == 0
