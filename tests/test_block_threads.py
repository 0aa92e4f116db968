"""The block size a caller asks for (csrc/wavefront.h block_threads): k_primary deals image tiles to whole warps, so
every count becomes a multiple of 32 from 32 to 256.  The rule is compiled and run on the host."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import bit_mismatches

ROOT = Path(__file__).resolve().parent.parent

SRC = """
#include <cstdio>
#include "wavefront.h"
int main()
{
    for (int t = -40; t <= 1100; ++t) std::printf("%d %d\\n", t, atx::block_threads(t));
}
"""


def test_blocks_are_whole_warps(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'ataraxia_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    f"-I{cuda / 'include'}", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    for line in out.splitlines():
        asked, got = map(int, line.split())
        assert got % 32 == 0 and 32 <= got <= 256
        if 32 <= asked <= 256:
            assert got == asked - asked % 32
        elif asked <= 0 or asked > 256:
            assert got == 256


@pytest.mark.gpu
@pytest.mark.parametrize("bvh", [False, True])
def test_any_count_renders_the_same(po, bvh):
    from ataraxia_gb300 import Renderer, Settings, scenes

    sc = scenes.config1().with_resolution(321, 97)
    view = po.view_for(sc)

    def frames(threads):
        with Renderer(threads=threads, bvh_threshold=2 if bvh else 0, hbm_budget_bytes=4 << 30) as r:
            r.on_resize(sc.width, sc.height)
            r.set_scene(sc.spheres, sc.materials, sc.lights)
            r.set_camera_matrices(np.array(view.inv_view), np.array(view.inv_proj), sc.camera_position)
            r.set_settings(Settings(accumulation=True, skyLight=False, maxBounces=4))
            r.render_frames(1)   # without the per-camera tables
            r.render_frames(6)
            return r.get_accumulation()

    want = frames(0)
    for threads in (1, 31, 32, 48, 100, 255, 256, 300):
        assert bit_mismatches(frames(threads), want) == 0, threads
