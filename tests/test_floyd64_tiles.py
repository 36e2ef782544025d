"""The tiles that the CTAs of the blocks-of-64 Floyd remainder take
(floyd64_tiles.h, compiled for the host): every tile has one writer, directly or
as the transpose of its mirror image."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastapsp_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "floyd64_tiles.h"
int main() {
  for (int sym = 0; sym < 2; sym++)
    for (int nr = 1; nr < 24; nr++) {
      std::vector<int> writers(nr * nr, 0);
      for (int jx = 0; jx < nr; jx++)
        for (int i0 = 0; i0 < nr; i0 += 2)
          for (int i = i0; i < i0 + fapb::floyd64_pair_rows(sym, jx, i0, nr); i++) {
            if (i >= nr) return std::printf("row %d of %d\n", i, nr), 1;
            writers[i * nr + jx]++;
            if (sym && i != jx) writers[jx * nr + i]++;
          }
      for (int t = 0; t < nr * nr; t++)
        if (writers[t] != 1) return std::printf("sym %d nr %d tile (%d, %d): %d writers\n", sym, nr, t / nr, t % nr, writers[t]), 1;
    }
  return 0;
}
"""


def test_every_tile_has_one_writer(tmp_path):
    src = tmp_path / "tiles.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "tiles"
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
