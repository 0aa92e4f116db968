"""Whole paths in one thread for small waves (csrc/wavefront.cu k_fused, wavefront.h kFusedSmallWork)."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [25, 64, 65])
def test_small_waves_in_one_thread_bit_exact(po, n):
    """Up to 64 spheres in waves small enough for whole paths in one thread, and one sphere past them."""
    st = scenes.Stream(43, f"small{n}")
    s = scenes._spheres(st.uniform(3 * n, -8, 8).reshape(n, 3), st.lognormal(0.0, 0.4, n), st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 5.0, 22.0))
    sc = scenes.SyntheticScene("small", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, 3, 14.0), pos, d,
                               width=67, height=29, max_bounces=7)
    view = po.view_for(sc)
    for spp in (1, 3, 8, 9):
        with Renderer() as r:
            r.on_resize(sc.width, sc.height)
            r.set_scene(sc.spheres, sc.materials, sc.lights)
            r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
            r.set_settings(Settings(maxBounces=7))
            r.render_frames(spp)
            got = r.get_accumulation().reshape(-1, 4)
        want, _, _ = oracle_render(sc, spp)
        assert bit_mismatches(got, want) == 0
