"""The base-256 digits of the split-precision slicer (green-mbpt_b200/csrc/split_digits.cuh), compiled as host code:
for every slice count 2..6 and values across the whole range |X| <= 2^(8S-2), ends included, the digits of X and of -X
are those of the bottom-up construction (lower ones in [-128, 127], the top one at most 64), and rebuild the value."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r'''
#include <cstdio>
#include "split_digits.cuh"
int main() {
  int S; double x;
  while (std::scanf("%d %lf", &S, &x) == 2) {
    const unsigned long long u = gb200::wide_input(x, S), v = gb200::wide_negate(u, S);
    for (int s = 0; s < S; ++s) {
      const unsigned w = gb200::wide_digit_word(u, v, u, v, S, s);
      std::printf("%d %d ", (int)(signed char)(w & 0xFF), (int)(signed char)((w >> 8) & 0xFF));
    }
    std::printf("\n");
  }
  return 0;
}
'''


def bottom_up(X, S):
    d = []
    for _ in range(S - 1):
        r = ((X + 128) % 256) - 128
        d.append(r)
        X = (X - r) // 256
    return [X] + d[::-1]


def test_wide_digits_match_bottom_up_construction(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not installed")
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "green-mbpt_b200", "csrc"),
                        str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(0)
    cases = []
    for S in range(2, 7):
        lim = 1 << (8 * S - 2)
        vals = [0, 1, -1, 127, 128, -128, -129, 255, 256, lim, -lim, lim - 1, lim // 2] + [int(x) for x in rng.integers(-lim, lim, 200)]
        cases += [(S, v) for v in vals]
    r = subprocess.run([str(exe)], input="\n".join(f"{S} {v}" for S, v in cases), capture_output=True, text=True)
    lines = r.stdout.strip().splitlines()
    assert r.returncode == 0 and len(lines) == len(cases)
    for (S, v), line in zip(cases, lines):
        got = [int(x) for x in line.split()]
        assert got[0::2] == bottom_up(v, S) and got[1::2] == bottom_up(-v, S), (S, v)
        assert abs(got[0]) <= 64 and abs(got[1]) <= 64
