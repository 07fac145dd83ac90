"""Where the PME spread writes a grid point (caps_b200/csrc/pme.cuh, grid_cell), compiled for the host: grids up to past 2^31
points, as long as a line transform can be along one axis."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
SOURCE = """
#include <cstdio>
#include "pme.cuh"
int main() {
  int k1, k2, a, b, c;
  while (std::scanf("%d %d %d %d %d", &k1, &k2, &a, &b, &c) == 5) std::printf("%zu\\n", capsb::grid_cell(a, b * k1, c, k1 * k2));
}
"""


@pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")
def test_grid_cell_past_32_bits(tmp_path):
    (tmp_path / "cell.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "caps_b200" / "csrc"),
                    str(tmp_path / "cell.cu"), "-o", str(tmp_path / "cell")], check=True)
    asked = []
    for k in [(9, 10, 12), (70, 70, 70), (1280, 1296, 1280), (1296, 1296, 1296), (4800, 700, 800), (27, 9600, 9600)]:
        for p in [(0, 0, 0), (k[0] - 1, 0, 0), (0, k[1] - 1, 0), (0, 0, k[2] - 1), tuple(n - 1 for n in k), tuple(n // 2 for n in k)]:
            asked.append((k, p))
    text = "\n".join(f"{k[0]} {k[1]} {p[0]} {p[1]} {p[2]}" for k, p in asked)
    got = subprocess.run([str(tmp_path / "cell")], input=text, capture_output=True, text=True, check=True).stdout.split()
    for (k, p), g in zip(asked, got):
        assert int(g) == p[0] + k[0] * (p[1] + k[1] * p[2]), (k, p)
    assert max(int(g) for g in got) > 2 ** 31
