"""Light and direction buffers of LBVH scenes (SceneStore::build_lists): once a scene has traced enough paths
its rays go through the cell lists, with the walk for cells that overflowed.  Frames before and after equal the
general path (brute force over the whole table) bit for bit."""
import numpy as np
import pytest

from helpers import bit_mismatches
from ataraxia_gb300 import Batch, Camera, Renderer, Settings, scenes
from ataraxia_gb300 import _native

pytestmark = pytest.mark.gpu


def _scene(kind, n, lights):
    st = scenes.Stream(23, f"lists{kind}{n}")
    half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
    c = st.uniform(3 * n, -half, half).reshape(n, 3)
    if kind == "clump":   # most cells of the spheres inside overflow
        c[: n // 2] *= 0.08
    if kind == "tied":    # every sphere twice: ties on t go to the lower index
        c[n // 2:2 * (n // 2)] = c[: n // 2]
    r = st.lognormal(-0.5, 0.5, n)
    if kind == "tied":
        r[n // 2:2 * (n // 2)] = r[: n // 2]
    lt = scenes.draw_lights(st, lights, 1.5 * half)
    if lights > 1:
        lt["position"][0] = (0.1, 0.2, 0.3)   # one in the middle of the spheres
    pos, d = scenes._look_at((0.0, 0.6 * half, 2.0 * half))
    return scenes.SyntheticScene(kind, scenes._spheres(c, r, st.integers(0, 16, n)), scenes.draw_materials(st, 16), lt,
                                 pos, d, far=1000.0, width=127, height=61, max_bounces=6)


def _render(sc, calls, sky, **kw):
    out = []
    with Renderer(**kw) as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
        r.set_settings(Settings(accumulation=True, skyLight=sky, maxBounces=sc.max_bounces))
        for spp in calls:
            r.render_frames(spp)
            out.append(r.get_accumulation().reshape(-1, 4).copy())
        return out, r.stats()["device_bytes"]


# the smallest LBVH scene, one in between and the most spheres with lists; the calls' paths pass
# 2 n^2 with the second call
@pytest.mark.parametrize("kind,n,lights,sky", [("open", 1025, 1, False), ("clump", 1300, 5, True),
                                               ("tied", 1401, 40, False), ("open", 4096, 8, False),
                                               ("clump", 8192, 3, False)])
@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_RENDERS])
def test_lists_render_as_the_general_path(kind, n, lights, sky, flags):
    sc = _scene(kind, n, lights)
    frames = 2 * n * n // sc.pixels
    calls = (1, frames, 3, 1)
    want, small = _render(sc, calls, sky, bvh_threshold=1 << 30)
    got, large = _render(sc, calls, sky, flags=flags)
    assert large > n * 300_000          # the lists were built
    for a, b in zip(got, want):
        assert bit_mismatches(a, b) == 0


def test_lists_wait_for_enough_paths_and_for_memory():
    sc = _scene("open", 1025, 3)
    frames = 2 * 1025 * 1025 // sc.pixels + 1
    _, few = _render(sc, (1, 2), False)
    assert few < 1025 * 300_000
    want, _ = _render(sc, (1, frames, 2), False, bvh_threshold=1 << 30)
    with_lists, large = _render(sc, (1, frames, 2), False)
    got, held = _render(sc, (1, frames, 2), False, hbm_budget_bytes=2_000_000_000)   # a budget: the tree, as before
    assert large > held + 1025 * 300_000
    for a, b, c in zip(got, with_lists, want):
        assert bit_mismatches(a, c) == 0 and bit_mismatches(b, c) == 0


def test_lists_in_a_batch_and_after_a_new_scene():
    a, b = _scene("open", 1100, 4), _scene("clump", 1200, 4)
    frames = 2 * 1200 * 1200 // a.pixels + 1
    with Batch() as bt:
        ids = [bt.add_synthetic(s) for s in (a, b)]
        for spp in (2, frames, 2, 2):   # the same shape again: the pass becomes a graph
            for i in ids:
                bt.set_spp(i, spp)
            bt.run()
        got = [bt.get_accumulation(i) for i in ids]
    for s, g in zip((a, b), got):
        want, _ = _render(s, (2, frames, 2, 2), False, bvh_threshold=1 << 30)
        assert bit_mismatches(g, want[-1]) == 0
    with Renderer() as r:               # lists of one scene are not used for the next
        for s in (a, b, a):
            r.on_resize(s.width, s.height)
            r.set_scene(s.spheres, s.materials, s.lights)
            r.set_camera(Camera(s.fov, s.near, s.far, s.camera_position, s.camera_direction))
            r.set_settings(Settings(maxBounces=s.max_bounces))
            r.reset_frame_index()
            for spp in (1, frames, 1):
                r.render_frames(spp)
            got = r.get_accumulation().reshape(-1, 4)
            want, _ = _render(s, (1, frames, 1), False, bvh_threshold=1 << 30)
            assert bit_mismatches(got, want[-1]) == 0


def _launches(r, spp=2):
    """Kernels of one render: six through the lists, five on the tree (waves this small)."""
    before = r.stats()["kernel_launches"]
    r.render_frames(spp)
    return r.stats()["kernel_launches"] - before


# a build of few and of many parts (4 M pairs of spheres a render of this size): every render in between on the tree
@pytest.mark.parametrize("kind,n,parts", [("open", 1025, 1), ("open", 4096, 4), ("clump", 8192, 16)])
@pytest.mark.parametrize("flags", [0, _native.FLAG_OVERLAP_RENDERS])
def test_lists_are_built_in_parts(kind, n, parts, flags):
    sc = _scene(kind, n, 5)
    calls = (1, 2 * n * n // sc.pixels + 1) + (2,) * (parts + 2)
    want, _ = _render(sc, calls, False, bvh_threshold=1 << 30)
    used = []
    with Renderer(flags=flags) as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
        r.set_settings(Settings(maxBounces=sc.max_bounces))
        for spp, w in zip(calls, want):
            used.append(_launches(r, spp))
            assert bit_mismatches(r.get_accumulation().reshape(-1, 4), w) == 0
    assert used[2:] == [5] * (parts - 1) + [6] * 3


def test_no_lists_for_rays_that_are_not_traced():
    n = 1100
    sc = _scene("open", n, 4)
    frames = 2 * n * n // sc.pixels + 1
    cam = Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction)
    away = Camera(sc.fov, sc.near, sc.far, sc.camera_position, tuple(-np.array(sc.camera_direction)))
    with Renderer(wave_paths=1 << 18) as r:   # little path state beside the lists
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_settings(Settings(maxBounces=1))
        r.set_camera(cam)
        for _ in range(3):                       # no bounce that would leave a sphere
            r.render_frames(frames)
        assert r.stats()["device_bytes"] < n * 300_000
        r.set_settings(Settings(maxBounces=sc.max_bounces))
        r.set_camera(away)
        for _ in range(6):                       # a camera that sees no sphere
            r.render_frames(frames)
        assert r.stats()["device_bytes"] < n * 300_000
        r.set_camera(cam)
        r.reset_frame_index()
        for _ in range(12):                      # and one that turns to them
            r.render_frames(frames)
        assert r.stats()["device_bytes"] > n * 300_000
        got = r.get_accumulation().reshape(-1, 4)
    want, _ = _render(sc, (frames,) * 12, False, bvh_threshold=1 << 30)
    assert bit_mismatches(got, want[-1]) == 0


def test_lists_are_given_back_for_a_smaller_scene():
    n = 2000
    big, half, small = _scene("open", n, 4), _scene("open", 1030, 4), _scene("open", 40, 4)
    frames = 2 * n * n // big.pixels + 1
    with Renderer(wave_paths=1 << 18) as r:
        r.on_resize(big.width, big.height)
        r.set_camera(Camera(big.fov, big.near, big.far, big.camera_position, big.camera_direction))
        r.set_settings(Settings(maxBounces=big.max_bounces))

        def show(sc):
            r.set_scene(sc.spheres, sc.materials, sc.lights)
            r.reset_frame_index()
            r.render_frames(1)
            return r.stats()["device_bytes"]

        def go_on():
            for _ in range(3):
                r.render_frames(frames)
            return r.stats()["device_bytes"]

        without = show(big)
        assert without < n * 300_000
        assert go_on() > n * 786_432
        assert show(big) > n * 786_432        # the same scene again: what its lists will need is kept
        assert go_on() > n * 786_432
        assert show(half) > n * 786_432       # as for one that needs half of it
        show(big)
        go_on()
        assert show(small) < without + 40 * 400_000   # a table's own buffers
        show(big)
        go_on()
        r.set_scene(half.spheres[:1000], half.materials, half.lights)   # a table, no tree
        assert r.stats()["device_bytes"] < n * 300_000


def test_lists_of_more_spheres_in_a_face_than_a_block_keeps():
    from test_cells_gpu import slab

    n = 4000
    sc = slab(n)
    calls = (1, 2 * n * n // sc.pixels + 1) + (2,) * 6
    want, _ = _render(sc, calls, True, bvh_threshold=1 << 30)
    with Renderer() as r:
        r.on_resize(sc.width, sc.height)
        r.set_scene(sc.spheres, sc.materials, sc.lights)
        r.set_camera(Camera(sc.fov, sc.near, sc.far, sc.camera_position, sc.camera_direction))
        r.set_settings(Settings(skyLight=True, maxBounces=sc.max_bounces))
        used = []
        for spp, w in zip(calls, want):
            used.append(_launches(r, spp))
            assert bit_mismatches(r.get_accumulation().reshape(-1, 4), w) == 0
    assert used[-1] == 6
