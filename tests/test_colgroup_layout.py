"""The column groups' arrays in shared memory (csrc/colgroup.cuh) are placed at
multiples of 16 bytes, so no element type may ask for more."""
import subprocess
from pathlib import Path

from parallellocallyoptimalapproximatesparsematrixinverses_b200 import build

PROGRAM = """
#include <cstdio>
#include "colgroup.cuh"
int main() {
  size_t window = 16;
  for (int words = 32; words <= 2048; words += 32) window = spai::WindowBytes(words) % 16 == 0 ? window : 0;
  std::printf("%zu %zu %zu %zu %zu\\n", window, alignof(spai::GroupValues<float, 2>), alignof(spai::GroupValues<float, 4>),
              alignof(spai::GroupValues<double, 2>), alignof(spai::GroupValues<double, 4>));
}
"""


def test_group_values_fit_their_places(tmp_path):
    source = tmp_path / "layout.cu"
    source.write_text(PROGRAM)
    program = tmp_path / "layout"
    subprocess.run([build.nvcc(), "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{build.CSRC}",
                    f"-I{Path(build.PACKAGE_DIR).parent / 'include'}", str(source), "-o", str(program)], check=True)
    window, *alignments = map(int, subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split())
    assert window == 16
    assert max(alignments) <= 16
