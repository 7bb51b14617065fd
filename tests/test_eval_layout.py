"""Shared memory of the evaluation kernel: every round of a search fits what its
launch allocates (host arithmetic of csrc/eval_layout.h, no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "eval_layout.h"
using namespace pgsvt;
int main() {
  int bad = 0, rounds = 0;
  for (int side = 2; side <= 16; ++side)
    for (int nwin = 1; nwin <= 21; nwin += 2) {
      const int bs = side <= 8 ? side : 0;  // the kernel's form
      const int NC = nwin <= 10 ? 10 : (nwin <= 16 ? 16 : 22);
      for (int wide = 0; wide < 2; ++wide)
        for (int points = 1; points <= 16; ++points) {
          const int words = eval_alloc_words(bs, wide, NC, nwin, points);
          for (int nl = 1; nl <= points; ++nl, ++rounds) {
            const int T = eval_tile(bs, wide, eval_large_rounds(bs, wide, NC, nwin, points), nl);
            // 16-byte clears of whole tiles; tiles large enough for one patch
            bool ok = T % 4 == 0 && T >= side * side && eval_tiles_at(bs, NC, nl) % 4 == 0;
            // the tiles are the last thing in the block's shared memory
            ok = ok && eval_tiles_at(bs, NC, nl) + nwin * 2 * T <= words;
            ok = ok && words * 4 <= 227 * 1024;
            if (wide) ok = ok && T == 256;  // rounding depends on the size
            if (points <= 8) ok = ok && T == eval_alloc_tile(bs, wide, 1);
            if (!ok && bad++ < 5)
              std::printf("side %d nwin %d wide %d points %d nl %d\n", side, nwin, wide, points, nl);
          }
        }
    }
  std::printf("%d rounds, %d bad\n", rounds, bad);
  return bad != 0;
}
"""


def test_every_round_fits_its_allocation(tmp_path):
    """A round of fewer lambda values than the launch allocates for (refinements
    place half of them, narrow searches fewer, the evaluation budget any number)."""
    src = tmp_path / "layout.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "layout"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "pgure-svt_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
