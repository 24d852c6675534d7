// bfvm_pair_coefs.h -- which chunks of a line's coefficient rows a ring of the
// paired sweeps (bfvm_pair_sweeps.cu) stages in shared memory.
//
// Plain arithmetic, without CUDA, so that a CPU test can hold every chunk
// against the room that the plan gives a ring.
#pragma once

#include "bfvm_host_device.h"

namespace bfvm {

// A line of n values in C chunks of R, whose rows are constant from entry
// `first` (AxisCoefs::conv) to entry n - 2: chunks k0 .. k1 hold one and the
// same pair of rows and are staged once.
struct PairConv {
  int k0, k1;  // none: k0 > k1
  BFVM_HD int sh() const { return k1 > k0 ? k1 - k0 : 0; }
  BFVM_HD int at(int c) const { return c < k0 ? c : (c - sh() > k0 ? c - sh() : k0); }
};

BFVM_HD PairConv pair_conv(int C, int R, int n, int first) {
  const int k0 = (first + R - 1) / R, k1 = (n - 1) / R - 1;  // chunks ending at n - 2 or before
  return n >= 3 && k1 >= k0 ? PairConv{k0, k1} : PairConv{C, C - 1};
}

// The same at a launch whose rings have room for the chunks of a line constant
// from entry `most`, the latest of the solve's substrates when the launch was
// planned.  A launch captured by the caller outlives the solve's rows
// (bfvm_set_fp64_chain computes new ones), so `first` may lie past it: such a
// launch's results mean nothing, but it stays within its rings.
BFVM_HD PairConv pair_conv(int C, int R, int n, int first, int most) {
  return pair_conv(C, R, n, first < most ? first : most);
}

}  // namespace bfvm
