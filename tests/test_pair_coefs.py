"""The coefficient chunks that a ring of the paired sweeps stages, on the CPU: at
most as many as it has room for, whatever the device's convergence index, and
each chunk of the line where its rows are."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "bfvm_pair_coefs.h"

int main() {
  for (int R : {16, 32})
    for (int n = 1; n <= 330; ++n) {
      const int C = (n + R - 1) / R;
      for (int most = 0; most <= n; ++most) {
        const int room = C - bfvm::pair_conv(C, R, n, most).sh();
        for (int first = 0; first <= n; ++first) {
          const bfvm::PairConv v = bfvm::pair_conv(C, R, n, first, most);
          bool ok = C - v.sh() <= room;
          for (int c = 0; c < C; ++c) {
            const int at = v.at(c);
            ok = ok && at >= 0 && at < C - v.sh();
            if (first > most) continue;
            // the rows staged at `at` are those of this chunk: its own, or
            // those of another that lies in the constant entries with it
            const int from = at > v.k0 ? at + v.sh() : at;
            ok = ok && (from == c || (c * R >= first && from * R >= first && (c + 1) * R - 1 <= n - 2 &&
                                      (from + 1) * R - 1 <= n - 2));
          }
          if (!ok) {
            std::printf("R %d n %d most %d first %d\n", R, n, most, first);
            return 0;
          }
        }
      }
    }
  return 0;
}
"""


def test_staged_chunks_fit_their_ring(tmp_path):
    src = tmp_path / "coefs.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "coefs"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "physicell-x_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out == ""
