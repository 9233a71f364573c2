"""Host-compilable parts of the device headers, checked on the CPU: the layout of the crystals' cells."""
import json
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "fgrain_gb300" / "csrc"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """Compiles and runs a program (nvcc, host code only, no contraction); its output is JSON."""
    nvcc = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"

    def go(name, text):
        d = tmp_path_factory.mktemp(name)
        (d / "main.cu").write_text(text)
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-Xcompiler", "-ffp-contract=off",
                        "-I", str(CSRC), "-o", str(d / "main"), str(d / "main.cu")], check=True, capture_output=True)
        return json.loads(subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout)

    return go


def test_every_coordinate_names_a_cell_of_its_axis(run):
    """cells_layout over boxes from a cube to a thread a million times as long as wide: the last cell's
    number is exact in float (a coordinate is clamped to it), the box's cells are numbered in 32 bits,
    and there are at most 8 n + 64 of them."""
    r = run("cells", r"""
#include <cstdio>
#include "fg_cells.cuh"
int main() {
  int bad = 0, boxes = 0;
  for (double len : {1e0, 1e2, 1e4, 1e6, 3e6, 1e7, 1e8})
    for (double side : {1.0, 7.0, 300.0})
      for (double n : {1.0, 1e3, 1e5, 3e6, 4.1e6, 2e7, 2.1e9})
        for (int axis = 0; axis < 3; ++axis) {
          fg::CellGrid g{};
          const double b[3] = {axis == 0 ? len : side, axis == 1 ? len : side, axis == 2 ? len : side};
          if (!fg::cells_layout(b[0], b[1], b[2], n, g)) { ++bad; continue; }
          ++boxes;
          const double cells = 1.0 * g.x.n * g.y.n * g.z.n;
          for (const fg::CellAxis* a : {&g.x, &g.y, &g.z})
            if (a->n < 1 || static_cast<double>(a->last) != a->n - 1.0) ++bad;
          if (cells > 8.0 * n + 64.0 || cells >= 4294967296.0) ++bad;
        }
  std::printf("{\"bad\": %d, \"boxes\": %d}\n", bad, boxes);
}
""")
    assert r["boxes"] == 7 * 3 * 7 * 3 and r["bad"] == 0
