"""Late bounces (csrc/wavefront.cu k_paths): a lane carries a path to its end and takes the next of its warp's
share.  Frames rendered in many lanes and one big wave equal those of small single waves bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Camera, Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


def _frames(sc, calls, sky, **kw):
    with Renderer(**kw) as r:
        r.on_resize(sc.width, sc.height)
        r.set_tuning(path_kernel=1)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
        r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=sc.max_bounces))
        for spp in calls:
            r.render_frames(spp)
        return r.get_accumulation()


# queues from a few paths (fewer than a warp, a warp less and more one) to many chunks for every warp; long
# brute-force traces between the warps' refills (2,000 spheres without cell lists) and short ones
@pytest.mark.parametrize("n,res,spp,bounces,threshold", [(40, (9, 5), 3, 15, 0), (256, (64, 36), 7, 3, 0),
                                                         (256, (640, 360), 40, 8, 0), (2000, (127, 61), 700, 6, 1 << 30)])
@pytest.mark.parametrize("sky", [False, True])
def test_waves_of_any_size_render_the_same(n, res, spp, bounces, threshold, sky):
    st = scenes.Stream(29, f"paths{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(0.2, 0.5, n), st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.0 * half))
    sc = scenes.SyntheticScene("paths", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, 5, 1.5 * half), pos, d,
                               far=1000.0, width=res[0], height=res[1], max_bounces=bounces)
    want = _frames(sc, (1, spp), sky, bvh_threshold=threshold, wave_paths=4096)
    for _ in range(2):
        assert bit_mismatches(_frames(sc, (1, spp), sky, bvh_threshold=threshold), want) == 0


# a ground sphere of radius 1000 under a few spheres, whose cell lists hold most of the table: 64 samples and up to
# 15 bounces on two lanes, each frame sum against the oracle, over and over
@pytest.mark.parametrize("bounces,sky", [(5, False), (15, True)])
def test_ground_scene_repeats_bit_exact(po, bounces, sky):
    sc = scenes.config0().with_resolution(640, 360)
    sc.max_bounces = bounces
    want, _, _ = oracle_render(sc, 64, sky=sky)
    view = po.view_for(sc)
    with Renderer() as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=bounces))
        for _ in range(20):
            r.reset_frame_index()
            r.render_frames(64)
            assert bit_mismatches(r.get_accumulation().reshape(-1, 4), want) == 0
            assert np.array_equal(r.get_image().reshape(-1), po.pack_rgba8(want, 64))
