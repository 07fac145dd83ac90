"""Where the PME spread writes a grid point (caps_b200/csrc/pme.cuh, grid_place), compiled for the host: grids up to past 2^31
points, as long as a line transform can be along one axis, and which of them take places of 64 bits."""
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
  int k3;
  while (std::scanf("%d %d %d %d %d %d", &k1, &k2, &k3, &a, &b, &c) == 6) {
    size_t wide = 0;
    int narrow = 0;
    const bool needs = capsb::grid_needs_64(k1, k2, k3);
    const int p[3] = {a, b, c};
    for (int d = 0; d < 3; ++d) wide += capsb::grid_place<size_t>(p[d], d, k1, k2);
    if (!needs)
      for (int d = 0; d < 3; ++d) narrow += capsb::grid_place<int>(p[d], d, k1, k2);
    std::printf("%d %zu %d\\n", int(needs), wide, narrow);
  }
}
"""


@pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")
def test_grid_cell_past_32_bits(tmp_path):
    (tmp_path / "cell.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(ROOT / "caps_b200" / "csrc"),
                    str(tmp_path / "cell.cu"), "-o", str(tmp_path / "cell")], check=True)
    asked = []
    for k in [(9, 10, 12), (70, 70, 70), (1280, 1296, 1280), (1296, 1296, 1296), (4800, 700, 800), (27, 9600, 9600), (1024, 1024, 2048),
              (1024, 1024, 2047), (7, 7, 7 ** 8)]:
        for p in [(0, 0, 0), (k[0] - 1, 0, 0), (0, k[1] - 1, 0), (0, 0, k[2] - 1), tuple(n - 1 for n in k), tuple(n // 2 for n in k)]:
            asked.append((k, p))
    text = "\n".join(" ".join(map(str, k + p)) for k, p in asked)
    got = subprocess.run([str(tmp_path / "cell")], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    for (k, p), line in zip(asked, got):
        needs, wide, narrow = map(int, line.split())
        at = p[0] + k[0] * (p[1] + k[1] * p[2])
        assert needs == (k[0] * k[1] * k[2] > 2 ** 31 - 1) and wide == at and (needs or narrow == at), (k, p)
    assert {line[0] for line in got} == {"0", "1"}
