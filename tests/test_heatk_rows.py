"""The heat-with-k(x) kernels' row offsets (heatk_rows.h) on the host, up to the widest row the solver accepts: rows of
2^30 nodes put the row below a thread's two 2^31 elements away."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "multigpu_advectiondiffusion_gb300" / "csrc"
MAIN = """
#include <cstdint>
#include <cstdio>
#include "heatk_rows.h"
template <int RY> void show(int y, int nx, int ny) {
  adv::HeatKRows<RY> r;
  r.set(y, nx, ny);
  for (int i = 0; i < RY; ++i) std::printf("%lld ", (long long)(int64_t)r.dr[i]);
  std::printf("%lld %lld\\n", (long long)(int64_t)r.above, (long long)(int64_t)r.below);
}
int main() {
  int y, nx, ny, ry;
  while (std::scanf("%d %d %d %d", &ry, &y, &nx, &ny) == 4) ry == 1 ? show<1>(y, nx, ny) : show<2>(y, nx, ny);
}
"""


def test_row_offsets(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "rows.cpp").write_text(MAIN)
    exe = tmp_path / "rows"
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "rows.cpp"), "-o", str(exe)],
                   check=True)
    cases = [(ry, y, nx, ny) for ry in (1, 2) for nx in (1, 5, 1 << 29, (1 << 30) - 4, 1 << 30) for ny in (1, 2, 3, 7)
             for y in range(ny)]
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), text=True, check=True,
                         capture_output=True).stdout
    for (ry, y, nx, ny), line in zip(cases, out.splitlines(), strict=True):
        row = lambda r: (min(y + r, ny - 1) - y) * nx  # noqa: E731
        assert [int(v) for v in line.split()] == [row(r) for r in range(ry)] + [-nx if y else 0, row(ry)]
