"""k_infect's list of a unit's rows (replay_b200/csrc/unit_rows.h) gives back
every row with its first pair and its number of pairs, up to the longest row a
window can hold: the countdown rule lists rows of any length.  On the host: a
window with such a row takes 2^24 contacts and more."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r'''
#include <cstdio>
#include "unit_rows.h"
int main() {
  static rp::UnitRows<true> u;
  static rp::UnitRows<false> g;
  const int32_t lens[] = {1, 2, 48, (1 << 24) - 1, 1 << 24, (1 << 24) + 1, (1 << 25) + 100, 1 << 30, INT32_MAX};
  const int k = sizeof(lens) / sizeof(lens[0]);
  for (int p = 0; p < rp::kUnitRows; ++p) u.put(p, rp::kUnitRows - 1 - p, INT32_MAX - p, lens[p % k]);
  for (int p = 0; p < rp::kUnitRows; ++p) {
    int r;
    int32_t first, pairs;
    u.get(p, r, first, pairs);
    if (r != rp::kUnitRows - 1 - p || first != INT32_MAX - p || pairs != lens[p % k]) {
      printf("row %d: %d %d %d\n", p, r, first, pairs);
      return 1;
    }
  }
  // geometric rows: the longer ones go another way (kHeavyPairs)
  for (int p = 0; p < rp::kUnitRows; ++p) g.put(p, rp::kUnitRows - 1 - p, INT32_MAX - p, 1 + p % 48);
  for (int p = 0; p < rp::kUnitRows; ++p) {
    int r;
    int32_t first, pairs;
    g.get(p, r, first, pairs);
    if (r != rp::kUnitRows - 1 - p || first != INT32_MAX - p || pairs != 1 + p % 48) return 1;
  }
  return 0;
}
'''


def test_rows_keep_their_length(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "rows.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "rows"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "replay_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
