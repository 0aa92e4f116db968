"""The dynamic shared memory limit of a kernel belongs to the process, not to a caller: scenes of different sizes, set
and rendered in turn or by threads of their own, do not lower one another's."""
import threading

import numpy as np
import pytest

from helpers import bit_mismatches
from ataraxia_gb300 import Camera, Renderer, Settings, scenes

pytestmark = pytest.mark.gpu


def _scene(n, lights=3):
    st = scenes.Stream(5, f"limits{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    s = scenes._spheres(st.uniform(3 * n, -half, half).reshape(n, 3), st.lognormal(-0.5, 0.5, n), st.integers(0, 8, n))
    pos, d = scenes._look_at((0.0, 0.6 * half, 3.0 * half))
    return scenes.SyntheticScene(f"limits{n}", s, scenes.draw_materials(st, 8), scenes.draw_lights(st, lights, 1.5 * half),
                                 pos, d, far=1000.0, width=64, height=36, max_bounces=4)


def _set(r, sc):
    r.on_resize(sc.width, sc.height)
    r.set_scene(sc.spheres, sc.materials, sc.lights)
    r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
    r.set_settings(Settings(accumulation=True, skyLight=False, maxBounces=sc.max_bounces))


def _frames(r, spp=4):
    r.reset_frame_index()
    r.render_frames(spp)
    return r.get_accumulation().copy()


# tables staged in 48 to 96 KB of shared memory (more lights than a light buffer holds, so the bounces test them whole):
# the smaller scene is planned last, then the larger one renders and traces
def test_a_smaller_scene_does_not_lower_a_larger_ones_limit():
    big, small = _scene(5600, 70), _scene(3300, 70)
    o = np.zeros((64, 3), dtype=np.float32)
    d = np.tile(np.array([[0.6, 0.0, 0.8]], dtype=np.float32), (64, 1))
    with Renderer(bvh_threshold=1 << 30) as a, Renderer(bvh_threshold=1 << 30) as b:
        _set(a, big)
        want, hit = _frames(a), a.trace_nearest(o, d)
        _set(b, small)
        _frames(b)
        b.trace_nearest(o, d)
        assert bit_mismatches(_frames(a), want) == 0
        assert np.array_equal(a.trace_nearest(o, d)[1], hit[1])


# whole paths in one thread over such a table
def test_fused_paths_take_a_large_table():
    sc = _scene(3300, 70)
    with Renderer(bvh_threshold=1 << 30) as r:
        _set(r, sc)
        want = _frames(r)
        r.set_tuning(path_kernel=2)
        assert bit_mismatches(_frames(r), want) == 0


# light buffers built by several threads at once, of tables above and below what their builds may use without a raised
# limit
def test_threads_build_cell_lists_of_different_sizes():
    errors = []

    def work(n):
        try:
            sc = _scene(n)
            with Renderer(bvh_threshold=1 << 30) as r:
                _set(r, sc)
                want = _frames(r)
                for _ in range(400):
                    r.set_scene(sc.spheres, sc.materials, sc.lights)
                if bit_mismatches(_frames(r), want):
                    raise AssertionError("frames differ")
        except Exception as e:   # noqa: BLE001
            errors.append(f"{n} spheres: {e}")

    todo = [threading.Thread(target=work, args=(n,)) for n in (2500, 1030, 2500, 1100, 1300, 1030)]
    for t in todo:
        t.start()
    for t in todo:
        t.join()
    assert not errors, errors
