"""Frame 1 starts the accumulator from zero without a clearing pass: stale contents never show, in waves of
several sample chunks, whole paths in one thread and wavefront stages, with and without bounces, lanes that run
on from one render to the next."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes
from ataraxia_gb300 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,wave", [(1, 0), (2, 0), (1, 300)])
@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_RENDERS])
def test_frame_one_starts_from_zero(po, kernel, wave, flags):
    sc = scenes.config0().with_resolution(53, 31)
    view = po.view_for(sc)
    with Renderer(flags=flags, wave_paths=wave) as r:
        r.on_resize(sc.width, sc.height)
        r.set_tuning(path_kernel=kernel, wave_paths=wave)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        for bounces, sky in ((5, True), (0, True), (2, False)):
            r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=bounces))
            r.reset_frame_index()
            for spp in (7, 2):      # frames 1..7 over whatever the accumulator holds, then 8 and 9
                r.render_frames(spp)
            got = r.get_accumulation().reshape(-1, 4)
            want, _, _ = oracle_render(sc, 9, max_bounces=bounces, sky=sky)
            assert bit_mismatches(got, want) == 0
        r.set_settings(Settings(accumulation=False, skyLight=True, maxBounces=3))   # every render is frames 1..spp
        for _ in range(3):
            r.render_frames(4)
        want, _, _ = oracle_render(sc, 4, max_bounces=3, sky=True)
        assert bit_mismatches(r.get_accumulation().reshape(-1, 4), want) == 0
