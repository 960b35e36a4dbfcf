"""The rules by which a host bound of the particle count sizes the pair launches,
run on the host: a launch and its partial buffers hold whatever live count the
kernels find at or below the bound."""
import subprocess
from pathlib import Path

import pytest

from bromoc_gb300 import build

SRC = Path(__file__).resolve().parents[1] / "bromoc_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "launch.h"
using namespace bgpu;
int bgpu::n3_wave() { return 16 * kSMs; }
int main() {
  for (int bound = 1; bound <= kN3MaxTiles; ++bound)
    for (int t = 1; t <= bound; ++t)
      if (n64_grid(bound) < n64_blocks(t)) {
        std::printf("FP64: bound of %d tiles, %d live: %d blocks for a stride of %d\n", bound, t,
                    n64_grid(bound), n64_blocks(t));
        return 1;
      }
  for (int wave : {0, n3_wave()})
    for (int bound = 1; bound <= kN3MaxTiles; ++bound)
      for (int t = 1; t <= bound; ++t) {
        const int s = n3_split_of(t, wave);
        if (n3_most_work(bound, wave) < n3_work(t, s) ||
            n3_entries(bound) < (size_t)n3_pairs(t) * s) {
          std::printf("FP32: bound of %d tiles, %d live in %d parts\n", bound, t, s);
          return 1;
        }
      }
  return 0;
}
"""


@pytest.fixture(scope="module")
def nvcc():
    try:
        return build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")


def test_blocks_cover_every_live_count(nvcc, tmp_path):
    src = tmp_path / "bounds.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "bounds"
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", f"-I{SRC}", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
