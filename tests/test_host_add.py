"""add_all_or_nothing (csrc/host_add.h), through which the class-level entry
points add to the caller's arrays, compiled for the host with a fetch that
copies from memory or fails at a piece: the whole sum or nothing, for sizes
around the piece and one to six threads."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "host_add.h"

int main() {
  const size_t piece = 8;
  int bad = 0;
  for (size_t n : {0, 1, 7, 8, 9, 16, 40, 43, 200}) {
    for (int slots = 1; slots <= 6; slots++) {
      const int pieces = (int)((n + piece - 1) / piece);
      for (int fail = -1; fail < pieces; fail++) {
        std::vector<double> src(n), old(n), dst(n), want(n), bufs(slots * piece);
        for (size_t i = 0; i < n; i++) {
          src[i] = 0.1 * i + 1.0;
          want[i] = dst[i] = 3.0 - 0.7 * i;
          if (fail < 0) want[i] += 0.3 * src[i];
        }
        const int code = qbx::add_all_or_nothing(
            n, piece, slots, 0.3, old.data(), dst.data(),
            [&](int slot, size_t first, size_t count, const double** x) {
              if ((int)(first / piece) % slots != slot) return 99;   // not this slot's
              if ((int)(first / piece) == fail) return 7;
              std::memcpy(&bufs[slot * piece], src.data() + first, count * sizeof(double));
              *x = &bufs[slot * piece];
              return 0;
            });
        if (code != (fail < 0 ? 0 : 7) || dst != want) {
          std::printf("n %zu slots %d fail %d: code %d\n", n, slots, fail, code);
          bad = 1;
        }
      }
    }
  }
  return bad;
}
"""


def test_whole_sum_or_nothing(tmp_path):
    src = tmp_path / "add.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "add")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread",
                    "-I" + os.path.join(ROOT, "qbox-public_b200", "csrc"), str(src), "-o", exe],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
