"""The lines that the runs of steps in one launch prefetch, on the CPU: every
address lies in the tile's own rows, and together they are the tile's lines."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <set>
#include "bfvm_prefetch_lines.h"

// 0 where the lanes' lines are exactly those that hold the tile's values.
template <int AXIS, int LINE>
int check(int nx, int ny, int nz, int S) {
  const int nxp = (nx + LINE - 1) / LINE * LINE;
  const int xt = (nx + 31) / 32, nm = AXIS == 0 ? 1 : (AXIS == 1 ? nz : ny);
  const int per_s = AXIS == 0 ? (ny * nz + 31) / 32 : xt * nm;
  for (int tile = 0; tile < per_s * S; ++tile) {
    std::set<long long> want, got;
    const int s = tile / per_s, q = tile - s * per_s;
    auto row = [&](long long k, long long j, int i0, int i1) {
      for (int i = i0; i < i1; i += LINE) want.insert(((s * (long long)nz + k) * ny + j) * nxp + i);
    };
    if (AXIS == 0) {
      for (int r = 32 * q; r < 32 * q + 32 && r < ny * nz; ++r) row(r / ny, r % ny, 0, nxp);
    } else {
      const int m = q / xt, i0 = q % xt * 32, i1 = i0 + 32 < nxp ? i0 + 32 : nxp;
      for (int l = 0; l < (AXIS == 1 ? ny : nz); ++l) row(AXIS == 1 ? m : l, AXIS == 1 ? l : m, i0, i1);
    }
    for (int lane = 0; lane < 32; ++lane) {
      const bfvm::PrefetchLines l = bfvm::prefetch_lines<AXIS, LINE>(nx, ny, nz, nxp, tile, lane);
      long long at = l.at;
      for (int k = lane; k < l.count; k += 32, at += l.step) got.insert(at);
    }
    if (got != want) return 1;
  }
  return 0;
}

int main() {
  const int shapes[][4] = {SHAPES};
  for (const auto& s : shapes) {
    const int bad = check<0, 16>(s[0], s[1], s[2], s[3]) + check<1, 16>(s[0], s[1], s[2], s[3]) +
                    check<2, 16>(s[0], s[1], s[2], s[3]) + check<0, 32>(s[0], s[1], s[2], s[3]) +
                    check<1, 32>(s[0], s[1], s[2], s[3]) + check<2, 32>(s[0], s[1], s[2], s[3]);
    if (bad) std::printf("%d x %d x %d x %d: %d\n", s[0], s[1], s[2], s[3], bad);
  }
  return 0;
}
"""

# Rows that end in the first and in the second 128-byte line of their last
# tile, whole tiles, one value and one row; last x tiles of fewer rows.
SHAPES = [(1, 1, 1, 1), (16, 5, 3, 2), (17, 33, 2, 1), (32, 7, 9, 2), (40, 36, 30, 3), (47, 31, 35, 2), (64, 3, 40, 1),
          (66, 65, 7, 2), (129, 2, 34, 2)]


def test_prefetched_lines_are_the_tiles_own(tmp_path):
    src = tmp_path / "lines.cpp"
    src.write_text(PROGRAM.replace("SHAPES", ", ".join("{%d, %d, %d, %d}" % s for s in SHAPES)))
    exe = tmp_path / "lines"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "physicell-x_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == ""
