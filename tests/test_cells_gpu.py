"""Light- and direction-buffer construction (csrc/light_buffer.cu) at the edges of its tiles: frames that
look every shadow and extension ray up in the cell lists equal the oracle's matched-order brute force
bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


def _scene(n, far_light):
    """n spheres at the medium scene's density; far_light: one light so far off that every sphere lies in
    one face of its cube."""
    st = scenes.Stream(11, f"cells{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    mats = scenes.draw_materials(st, 8)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(-0.5, 0.5, n),
                        st.integers(0, 8, n))
    lights = scenes.draw_lights(st, 1 if far_light else 5, 1.5 * half)
    if far_light:
        lights["position"] = [[0.5 * half, 20.0 * half, -half]]
    pos, d = scenes._look_at((0.0, 0.6 * half, 3.0 * half))
    return scenes.SyntheticScene(f"cells{n}", s, mats, lights, pos, d, far=1000.0, width=61, height=37, max_bounces=6,
                                 spp=3, frames=3)


# cells along an edge: whole tiles, a part of one in either direction, one cell left over; spheres: one, a
# warp less and more one, past a block, the most with a direction buffer, and more than a block keeps for a
# face (light buffer only: no direction buffer above 1,024)
@pytest.mark.parametrize("res,n", [(8, 33), (9, 31), (12, 257), (25, 100), (31, 300), (32, 1), (32, 1024), (16, 1500)])
def test_cell_lists_bit_exact(po, res, n):
    sc = _scene(n, n == 1500)
    view = po.view_for(sc)
    with Renderer(bvh_threshold=1 << 30) as r:
        r.on_resize(sc.width, sc.height)
        r.set_tuning(cell_res=res, path_kernel=1)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(accumulation=True, skyLight=False, maxBounces=sc.max_bounces))
        r.render_frames(sc.spp)
        assert r.tuning()["cell_res"] == res
        got = r.get_accumulation().reshape(-1, 4)
    want, _, _ = oracle_render(sc, sc.spp)
    assert bit_mismatches(got, want) == 0


def slab(n):
    """n small spheres in a slab that fills one face of a light's cube above it, few to a cell: more than the 2,048 a
    block keeps for a face, and lists that hold (from 4,000 on also for the spheres at the slab's corners)."""
    st = scenes.Stream(13, f"slab{n}")
    c = np.stack([st.uniform(n, -34, 34), st.uniform(n, -2, 2), st.uniform(n, -34, 34)], axis=1)
    lights = scenes.draw_lights(st, 1, 10.0)
    lights["position"] = [[0.3, 38.0, -0.2]]
    pos, d = scenes._look_at((3.0, 30.0, 50.0))
    return scenes.SyntheticScene(f"slab{n}", scenes._spheres(c, st.uniform(n, 0.2, 0.6), st.integers(0, 8, n)),
                                 scenes.draw_materials(st, 8), lights, pos, d, far=1000.0, width=127, height=61,
                                 max_bounces=6, spp=3, frames=3)


def test_more_spheres_in_a_face_than_a_block_keeps(po):
    sc = slab(2500)
    view = po.view_for(sc)
    with Renderer(bvh_threshold=1 << 30) as r:
        r.on_resize(sc.width, sc.height)
        r.set_tuning(cell_res=32, path_kernel=1)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(accumulation=True, skyLight=False, maxBounces=sc.max_bounces))
        r.render_frames(sc.spp)
        assert r.tuning()["cell_res"] == 32
        got = r.get_accumulation().reshape(-1, 4)
    want, _, _ = oracle_render(sc, sc.spp)
    assert bit_mismatches(got, want) == 0
