"""The pieces of the PCG's asynchronous copies cover an array once and nothing beside it (csrc/copy_pieces.cuh)."""
from __future__ import annotations

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "andosim_b200" / "csrc"

PROGRAM = r"""
#include "copy_pieces.cuh"
#include <cstdio>
#include <vector>
int main() {
  for (int off = 0; off < 4; ++off)
    for (int n = 0; n <= 70; ++n) {
      std::vector<int> seen(n);
      const ando::CopyPieces p = ando::copy_pieces(off, n);
      if (p.head < 0 || p.head > 3 || p.tail < 0 || p.tail > 3 || p.head + p.tail > n) return std::printf("%d %d: %d, %d\n", off, n, p.head, p.tail) > 0;
      for (int e = 0; e < p.head; ++e) seen[e]++;
      for (int e = n - p.tail; e < n; ++e) seen[e]++;
      for (int q = p.q0; q < p.q1; ++q)
        for (int e = 4 * q - off; e < 4 * q - off + 4; ++e) {   // 16 bytes from a boundary on
          if (e < 0 || e >= n) return std::printf("%d %d: piece %d reads element %d\n", off, n, q, e) > 0;
          seen[e]++;
        }
      for (int e = 0; e < n; ++e)
        if (seen[e] != 1) return std::printf("%d %d: element %d copied %d times\n", off, n, e, seen[e]) > 0;
    }
  return 0;
}
"""


def test_pieces(tmp_path):
    src = tmp_path / "pieces.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "pieces"
    subprocess.run(["g++", "-std=c++17", "-x", "c++", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout

