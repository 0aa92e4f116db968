"""Primary hits by warp cones (csrc/wavefront.cu k_primary, k_tile_masks, k_tile_lists) where a warp's 32
pixels end one image row and start the next, with a moved camera (caps or the cone's walk) and with a camera
that stayed (tile masks or lists): frames equal the oracle bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


# rows of a few tiles and a rest, one short of a tile, narrower than a tile (a warp spans several rows), one
# pixel; up to 32 mask words, and tables past the staged caps; leaf clusters up to and past 16 spheres
@pytest.mark.parametrize("res", [(95, 11), (31, 23), (7, 30), (1, 5), (1281, 3)])
@pytest.mark.parametrize("n,threshold,leaf", [(40, 1 << 30, 0), (1024, 1 << 30, 0), (1100, 1 << 30, 0), (700, 1, 0),
                                              (700, 1, 24), (5, 1, 1)])
def test_rows_inside_a_warp_bit_exact(po, res, n, threshold, leaf):
    st = scenes.Stream(17, f"rows{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(0.0, 0.5, n), st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.0 * half))
    sc = scenes.SyntheticScene("rows", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, 3, 1.5 * half), pos, d,
                               width=res[0], height=res[1], max_bounces=2, spp=1)
    view = po.view_for(sc)
    with Renderer(bvh_threshold=threshold, bvh_leaf_size=leaf) as r:
        r.on_resize(*res)
        r.set_tuning(path_kernel=1, bvh_leaf_size=leaf)
        r.set_scene(s, sc.materials, sc.lights)
        r.set_settings(Settings(maxBounces=2))
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        for k in (1, 2, 1):   # the camera's tables are built on its second render
            r.render_frames(k)
        got = r.get_accumulation().reshape(-1, 4)
    want, _, _ = oracle_render(sc, 4)
    assert bit_mismatches(got, want) == 0
