"""Late bounces of LBVH scenes in one launch (csrc/wavefront.cu k_paths_walk, started at bounce 1 to 4 by the
wave's paths): frames equal the oracle, and waves that start it at different bounces each other, bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


def _scene(n, res, bounces, lights):
    st = scenes.Stream(37, f"walked{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(0.3, 0.5, n), st.integers(0, 8, n))
    m = scenes.draw_materials(st, 8)
    m["emission_color"][2] = 1.0
    m["emission_intensity"][2] = 0.5
    pos, d = scenes._look_at((0.0, 0.6 * half, 1.5 * half))
    return scenes.SyntheticScene("walked", s, m, scenes.draw_lights(st, lights, 1.5 * half), pos, d, far=1000.0,
                                 width=res[0], height=res[1], max_bounces=bounces)


def _frames(sc, view, spp, sky, **kw):
    with Renderer(bvh_threshold=1, **kw) as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=sc.max_bounces))
        r.render_frames(spp)
        return r.get_accumulation().reshape(-1, 4), r.stats()


# a path or two, a warp less and more one, no lights and more than a word of them, one bounce to many
@pytest.mark.parametrize("res,bounces,lights", [((2, 1), 15, 3), ((11, 3), 4, 0), ((61, 37), 2, 40), ((61, 37), 9, 8)])
@pytest.mark.parametrize("sky", [False, True])
def test_small_waves_bit_exact(po, res, bounces, lights, sky):
    sc = _scene(300, res, bounces, lights)
    got, _ = _frames(sc, po.view_for(sc), 3, sky)
    want, _, _ = oracle_render(sc, 3, sky=sky)
    assert bit_mismatches(got, want) == 0


def test_every_start_renders_the_same(po):
    sc = _scene(900, (640, 360), 6, 5)
    view = po.view_for(sc)
    # waves of at most 2^17, 2^20, 2^22 - and of all 4.6 M paths
    out = [_frames(sc, view, 20, True, wave_paths=w) for w in (1 << 17, 1 << 20, 1 << 22, 1 << 23)]
    for acc, st in out[1:]:
        assert st["shaded_first"] == out[0][1]["shaded_first"]
        assert bit_mismatches(acc, out[0][0]) == 0


# waves large enough that k_bounce's blocks gather hits over several turns of their share of the queue
# (bounces 1 to 3; a budget keeps the scene on its tree), against waves small enough to go without it;
# repeated, since warps that disagreed about a turn would differ from run to run
@pytest.mark.parametrize("spp", [24, 76])   # 5.5 M paths in one lane, 17.5 M in four
def test_gathered_bounces_repeat(po, spp):
    sc = _scene(1200, (640, 360), 5, 5)
    view = po.view_for(sc)
    want, _ = _frames(sc, view, spp, True, wave_paths=1 << 17, hbm_budget_bytes=8 << 30)
    with Renderer(bvh_threshold=1, hbm_budget_bytes=8 << 30) as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(accumulation=True, skyLight=True, maxBounces=sc.max_bounces))
        for _ in range(20):
            r.reset_frame_index()
            r.render_frames(spp)
            assert bit_mismatches(r.get_accumulation().reshape(-1, 4), want) == 0
