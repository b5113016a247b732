"""Four-row folding of the FP32 transforms (csrc/fold.hpp), compiled with g++ and
checked on the CPU.

Over the base rows of a geometry every row must be folded exactly once, at its own centred
coordinate (FT_r2c_padded's centring, litho.cpp:242-318), and the signs of the folding must give
that row's cos and sin from the base row's.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fpga-litho-accel_gb300", "csrc")

DRIVER = r"""
#include "fold.hpp"
#include <cmath>
#include <cstdio>
#include <vector>
using namespace litho;
static int rows(int L, int F) {
  std::vector<int> seen(L, 0);
  const int nb = fold_nbase(L, F), h = F / 2;
  const double w = 2 * M_PI / F;
  for (int b = 0; b < nb; ++b)
    for (int k = 0; k < 4; ++k) {
      const int Y = fold_row(b, k, L, F);
      const FoldRange r = fold_range(k, L, F);
      const bool in = (unsigned)(b - r.lo) < (unsigned)r.n;
      if (in != (Y >= 0)) { std::printf("range %d %d b %d k %d\n", L, F, b, k); return 1; }
      if (Y < 0) continue;
      if (Y >= L || fold_y(b, k, L, F) != Y) { std::printf("row %d %d b %d k %d\n", L, F, b, k); return 1; }
      const int yp = Y + fo_oy(L, F);
      if (yp != (k == 0 ? b : k == 1 ? -b : k == 2 ? h - b : b - h)) { std::printf("coord\n"); return 1; }
      for (int v = 0; v <= 5; ++v) {  // (even, odd) signs of the folded operands
        const double sg = v & 1 ? -1 : 1, c = std::cos(w * v * b), s = std::sin(w * v * b);
        const double ec = k < 2 ? c : sg * c, es = (k & 1 ? -1 : 1) * (k < 2 ? s : -sg * s);
        if (std::fabs(std::cos(w * v * yp) - ec) > 1e-9 || std::fabs(std::sin(w * v * yp) - es) > 1e-9) {
          std::printf("sign %d %d b %d k %d v %d\n", L, F, b, k, v);
          return 1;
        }
      }
      seen[Y]++;
    }
  for (int Y = 0; Y < L; ++Y)
    if (seen[Y] != 1) { std::printf("seen %d %d %d %d\n", L, F, Y, seen[Y]); return 1; }
  return 0;
}
int main() {
  int L, F;
  while (std::scanf("%d %d", &L, &F) == 2)
    if (rows(L, F)) return 1;
  std::printf("ok\n");
  return 0;
}
"""


def _pow2(n):
    p = 1
    while p < n:
        p *= 2
    return p


def test_every_row_folded_once(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "drv.cpp", tmp_path / "drv"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    lines = [f"{n} {f * _pow2(n)}" for n in range(2, 401) for f in (1, 2, 4)]
    lines += [f"{n} {_pow2(n)}" for n in (1024, 1025, 2048, 4096, 16384)]
    r = subprocess.run([str(exe)], input="\n".join(lines) + "\n", capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
