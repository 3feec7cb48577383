"""The split of a 1D solve over the blocks of its step loop's cluster, for every
length the loop takes: the blocks hold all points, and none is empty.  A block
without points sends nothing at the end of a step, so nothing would hold the
other blocks' next messages back until it has read the last ones."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "phasefield5d_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "pf5d_loop1d.h"
int main() {
  using namespace pf5d;
  for (int most : {16, 8})
    for (int64_t n = 1; n <= kLoop1dMax; ++n) {
      const Loop1dShape L = loop1d_shape(n, most);
      const bool ok = L.blocks >= 1 && L.blocks <= most && most <= kLoop1dBlocks &&
                      L.chunk % 32 == 0 && (int64_t)L.blocks * L.chunk >= n &&
                      (int64_t)(L.blocks - 1) * L.chunk < n && L.threads % 32 == 0 &&
                      L.threads >= 64 && L.threads <= kLoop1dThreads && 4 * L.blocks <= L.threads;
      if (!ok) {
        printf("n %lld most %d: %d blocks of %d points, %d threads\n", (long long)n, most, L.blocks,
               L.chunk, L.threads);
        return 1;
      }
    }
  return 0;
}
"""


def test_every_block_holds_points(tmp_path):
    src, exe = tmp_path / "shape.cpp", tmp_path / "shape"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
