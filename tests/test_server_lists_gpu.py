"""A served LBVH job that traces enough paths gets cell lists when it is admitted, within half of the budget:
its results equal the brute-force renderer's bit for bit, with lists and without."""
import numpy as np
import pytest

from ataraxia_gb300 import Camera, Renderer, Server, Settings, scenes
from tests.helpers import bit_mismatches

pytestmark = pytest.mark.gpu

N, SPP = 1100, 96          # 1100 spheres: lists from 4 * 1100^2 = 4.84 M paths on
LISTS = N * 6 * 32 * 32 * 64 * 2   # bytes of the direction buffer's cells


def _scene():
    st = scenes.Stream(5, "served lists")
    half = 32.0
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.0 * half))
    return scenes.SyntheticScene("served", scenes._spheres(st.uniform(3 * N, -half, half).reshape(N, 3),
                                                           st.lognormal(-0.5, 0.5, N), st.integers(0, 16, N)),
                                 scenes.draw_materials(st, 16), scenes.draw_lights(st, 4, 1.5 * half), pos, d,
                                 far=1000.0, width=257, height=199, max_bounces=6)


@pytest.mark.parametrize("spp,budget,lists", [(SPP, 0, True), (SPP, 3 * LISTS, True), (SPP, LISTS, False),
                                              (16, 0, False)])
def test_served_lists(spp, budget, lists):
    sc = _scene()
    with Server(hbm_budget_bytes=budget, pass_spp=8) as s:
        ids = [s.submit(sc, spp), s.submit(sc, 4)]
        peak = 0
        while s.stats()["completed"] < 2:
            peak = max(peak, s.stats()["device_bytes"])
        got = [(s.accumulation(j), s.image(j)) for j in ids]
        assert s.stats()["device_bytes"] < (1 << 20)
    assert (peak > LISTS) == lists
    for (acc, img), k in zip(got, (spp, 4)):
        with Renderer(bvh_threshold=1 << 30) as r:
            r.on_resize(sc.width, sc.height)
            r.set_scene(sc.spheres, sc.materials, sc.lights)
            r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
            r.set_settings(Settings(accumulation=True, skyLight=sc.sky_light, maxBounces=sc.max_bounces))
            r.render_frames(k)
            assert bit_mismatches(acc, r.get_accumulation().reshape(-1, 4)) == 0
            assert np.array_equal(img, r.get_image().reshape(-1))
