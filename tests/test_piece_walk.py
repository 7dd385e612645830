"""The walk over rows and pieces of the streaming passes (csrc/piece_walk.cuh), compiled for the host: every piece is taken once, and where the rows of a call end
near 2^31 the places behind them are behind them for the threads too."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "nano-qwen3tts-vllm_b200" / "csrc"
MAIN = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "piece_walk.cuh"
using namespace b2;
int main() {
  std::mt19937 r(7);
  for (int n = 0; n < 300; ++n) {                   // small calls: who takes what
    const int pieces = 1 + r() % (n % 3 ? 40 : 900), rows = 1 + r() % 60;
    const unsigned stride = 1 + r() % (n % 2 ? 70 : 5000);
    std::vector<int> taken(static_cast<size_t>(rows) * pieces, 0);
    const PieceStep s = piece_step(stride, pieces);
    for (unsigned i = 0; i < stride; ++i)
      for (PieceWalk w = piece_at(i, pieces); w.row < rows; w = piece_next(w, s, pieces)) {
        if (w.row < 0 || w.piece < 0 || w.piece >= pieces) return 1;
        ++taken[w.row * pieces + w.piece];
      }
    for (int t : taken) if (t != 1) return 2;
  }
  // the last places of the largest calls, reached from a few steps before them: rows of 8, 16, 96 and 2^31 - 8 columns, as many as an int counts
  const unsigned stride = 2368 * 256;
  for (int pieces : {1, 2, 12, 268435455}) {
    const int64_t rows = 2147483647, all = rows * pieces;
    const PieceStep s = piece_step(stride, pieces);
    for (unsigned i = 0; i < stride; i += 997) {
      int64_t flat = all - 5 * static_cast<int64_t>(stride) + i;
      PieceWalk w = {flat / pieces, static_cast<int>(flat % pieces)};
      for (int k = 0; k < 9; ++k) {
        if (w.row != flat / pieces || w.piece != flat % pieces || (w.row < rows) != (flat < all)) return 3;
        w = piece_next(w, s, pieces);
        flat += stride;
      }
    }
  }
  std::puts("ok");
}
"""


def test_every_piece_once_and_none_behind_the_last(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    assert subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout.split() == ["ok"]
