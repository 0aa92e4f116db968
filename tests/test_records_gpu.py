"""First bounce from per-pixel records and upload-time material rows (csrc/wavefront.cu PixelRecord,
make_material): materials at the edges of what the rows hold, and the smallest waves with records, equal the
oracle bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches, oracle_render
from ataraxia_gb300 import Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


def _scene():
    """Materials whose rows carry flags beside small or odd values: roughness 0 and below, metallic 0 to 1 in
    between and negative, emission on, off and negative, black and over-white albedo (roulette at 0.1 and 1)."""
    st = scenes.Stream(41, "records")
    rough = [0.0, -1.0, 1e-4, 1.0, 0.3, 0.05, 2.0, 0.5]
    metal = [0.0, 1.0, 0.5, -0.5, 1e-9, 1.0, 0.0, 0.25]
    glow = [0.0, 1.0, -1.0, 0.0, 3.0, 0.0, 1e-30, 0.5]
    m = scenes.draw_materials(st, 64)
    k = np.arange(64)
    m["roughness"] = np.float32(rough)[k % 8]
    m["metallic"] = np.float32(metal)[(k // 8) % 8]
    m["emission_color"] = st.uniform(192).reshape(64, 3)
    m["emission_intensity"] = np.float32(glow)[(k * 5) % 8]
    m["albedo"][k % 16 == 3] = 0.0
    m["albedo"][k % 16 == 7] = 1.5
    n = 200
    s = scenes._spheres(st.uniform(3 * n, -12, 12).reshape(n, 3), st.lognormal(0.2, 0.4, n), st.integers(0, 64, n))
    pos, d = scenes._look_at((0.0, 8.0, 30.0))
    return scenes.SyntheticScene("records", s, m, scenes.draw_lights(st, 7, 20.0), pos, d, width=61, height=37,
                                 max_bounces=5, spp=1)


# one sample (no records), two and three (the least slots a record has), a prime, a power of two; whole paths in
# one thread (k_fused) as well; the LBVH without lists (records, shadow rays of later bounces queued)
@pytest.mark.parametrize("spp", [1, 2, 3, 13, 16])
@pytest.mark.parametrize("kernel,threshold", [(1, 1 << 30), (2, 1 << 30), (1, 1)])
@pytest.mark.parametrize("bounces", [1, 5])
def test_records_and_material_rows_bit_exact(po, spp, kernel, threshold, bounces):
    sc = _scene()
    view = po.view_for(sc)
    with Renderer(bvh_threshold=threshold) as r:
        r.on_resize(sc.width, sc.height)
        r.set_tuning(path_kernel=kernel)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
        r.set_settings(Settings(maxBounces=bounces))
        r.render_frames(spp)
        got = r.get_accumulation().reshape(-1, 4)
    want, _, _ = oracle_render(sc, spp, max_bounces=bounces)
    ok = np.isfinite(want).all(1)   # black albedo and roughness -1 divide zero by zero: NaN wherever the oracle has it
    assert ok.mean() > 0.9
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert bit_mismatches(got[ok], want[ok]) == 0
