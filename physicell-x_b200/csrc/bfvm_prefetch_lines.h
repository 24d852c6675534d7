// bfvm_prefetch_lines.h -- the 128-byte lines of a 32-line tile, as the runs of
// steps in one launch (bfvm_resident.cu) ask for them ahead of the tile.
//
// Plain arithmetic, without CUDA, so that a CPU test can hold every address
// against the field's extent.
#pragma once

#include "bfvm_host_device.h"

namespace bfvm {

// Lane `lane`'s lines: elements at, at + step, at + 2 step, ... of the field,
// for the numbers q = lane, lane + 32, ... below count.
struct PrefetchLines {
  long long at, step;
  int count;
};

// Tile `tile` of the sweep along AXIS over a field of rows of nxp elements, a
// multiple of LINE, the elements of a 128-byte line.
template <int AXIS, int LINE>
BFVM_HD PrefetchLines prefetch_lines(int nx, int ny, int nz, int nxp, int tile, int lane) {
  PrefetchLines l;
  if (AXIS == 0) {
    const int rows = ny * nz, per_s = (rows + 31) / 32, s = tile / per_s, r0 = (tile - s * per_s) * 32;
    l.at = (static_cast<long long>(s) * rows + r0) * nxp + lane * LINE;
    l.step = 32 * LINE;
    l.count = (rows - r0 < 32 ? rows - r0 : 32) * (nxp / LINE);
  } else {
    constexpr int kLines = 32 / LINE;  // of the tile in a row
    const int nm = AXIS == 1 ? nz : ny, n = AXIS == 1 ? ny : nz;
    const int xt = (nx + 31) / 32, per_s = xt * nm, s = tile / per_s, q = tile - s * per_s, m = q / xt;
    const long long stride = AXIS == 1 ? nxp : static_cast<long long>(nxp) * ny;
    const long long plane = static_cast<long long>(s) * nz, row = AXIS == 1 ? (plane + m) * ny : plane * ny + m;
    const int i = (q - m * xt) * 32 + lane % kLines * LINE;
    l.at = row * nxp + i + lane / kLines * stride;
    l.step = 32 / kLines * stride;
    // (an FP64 row may end after the first line of its last tile: what follows
    // is the next row's, or past the field)
    l.count = i < nxp ? n * kLines : 0;
  }
  return l;
}

}  // namespace bfvm
