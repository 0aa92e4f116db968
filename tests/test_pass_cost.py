"""The batch's estimate of a scene's pass (csrc/batch_host.h pass_cost), compiled and run on the host: a ray through cell
lists or a table is cheaper than a walk of the tree they stand in for, by what they were measured to be."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

SRC = """
#include <cstdio>
#include "batch_host.h"
int main()
{
    for (unsigned n = 1; n <= 65536; n += n < 9000 ? 1 : 97)
        std::printf("%u %.9g %.9g\\n", n, atx::pass_cost(n, false, 1u << 24, 8), atx::pass_cost(n, true, 1u << 24, 8));
    std::printf("0 %.9g %.9g\\n", atx::pass_cost(9, false, 0, -3), atx::pass_cost(9, false, 0, 0));
}
"""


def test_lists_are_estimated_below_the_tree(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'ataraxia_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    f"-I{cuda / 'include'}", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    rows = [(int(n), float(a), float(b)) for n, a, b in (line.split() for line in out.splitlines())]
    assert rows[-1][1] == rows[-1][2] > 0.0          # no paths: a launch chain
    cost = {n: (a, b) for n, a, b in rows[:-1]}
    for n in range(1025, 8193):
        assert cost[n][0] < cost[n][1] / 3.0, n       # 1,025 to 8,000 spheres: measured 3.9 to 5.5 times
    keys = sorted(cost)
    assert all(cost[a][0] < cost[b][0] and cost[a][1] < cost[b][1] for a, b in zip(keys, keys[1:]))
