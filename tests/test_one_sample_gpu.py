"""Waves of one sample per pixel go through the shared primary hits (k_primary, then k_first over the hit
pixels): frames rendered one per call equal the oracle bit for bit, with the camera's tables and without."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


# warps whose pixels straddle tiles and the image's end; brute-force tables with and without lights, the LBVH
@pytest.mark.parametrize("n,res,lights,threshold", [(25, (33, 7), 4, 0), (256, (64, 36), 40, 0), (256, (31, 31), 0, 0),
                                                    (300, (45, 29), 8, 1)])
def test_one_sample_per_call_bit_exact(po, n, res, lights, threshold):
    st = scenes.Stream(5, f"one{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(0.0, 0.5, n),
                        st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.5 * half))
    sc = scenes.SyntheticScene("one", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, lights, 1.5 * half),
                               pos, d, width=res[0], height=res[1], max_bounces=5, spp=1)
    view = po.view_for(sc)
    with Renderer(bvh_threshold=threshold) as r:
        for sky in (False, True):
            r.on_resize(sc.width, sc.height)
            r.set_tuning(path_kernel=1)
            r.set_scene(sc.spheres, sc.materials, sc.lights)
            r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
            r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=sc.max_bounces))
            r.reset_frame_index()
            for _ in range(3):
                r.render_frames(1)
            got = r.get_accumulation().reshape(-1, 4)
            want, _, _ = oracle_render(sc, 3, sky=sky)
            assert bit_mismatches(got, want) == 0


def test_one_sample_statistics():
    sc = scenes.config1().with_resolution(160, 90)
    with Renderer() as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_settings(Settings(maxBounces=1))
        r.render_frames(1)
        st = r.stats()
        # one bounce: a primary ray per pixel, a shadow ray for every hit
        assert st["extension_rays"] == sc.pixels and st["shadow_rays"] == st["shaded_first"]
