"""Integer arithmetic of the kernels at the edge of its range (csrc/arith.cuh),
compiled for the host and run there: no GPU."""
from __future__ import annotations

import os
import subprocess

import pytest

from flashph_b200 import _build

SEARCH = r"""
#include <cstdio>
#include "arith.cuh"
// an ascending array of 2^31 - 2 entries that is not stored: entry p is p / 3
struct Entries {
  static constexpr long long N = (1ll << 31) - 2;
  mutable long long reads = 0, bad = 0;
  __host__ __device__ int operator[](long long p) const {
    ++reads;
    if (p < 0 || p >= N) ++bad;
    return (int)(p / 3);
  }
};
int main() {
  const int n = (int)Entries::N;
  const int ranges[][2] = {{0, 7}, {0, n}, {(1 << 30) - 9, (1 << 30) + 9}, {(1 << 30) + 5, n}, {n - 1, n}, {n - 40, n}};
  for (auto& r : ranges)
    for (int step = 0; step < 64; ++step) {
      const int at = (int)(r[0] + (long long)(r[1] - 1 - r[0]) * step / 63), x = at / 3;
      Entries a;
      const int got = ph::lower_bound_i32(a, r[0], r[1], x);
      const long long want = 3ll * x < r[0] ? r[0] : 3ll * x;
      if (a.bad || a.reads > 40 || got != want) {
        printf("[%d, %d) x %d: %d, not %lld; %lld reads, %lld outside\n", r[0], r[1], x, got, want, a.reads, a.bad);
        return 1;
      }
      const int mid = ph::midpoint(r[0], r[1]);
      if (mid < r[0] || mid >= r[1] || mid != ((long long)r[0] + r[1]) / 2) return 2;
    }
  return 0;
}
"""


@pytest.mark.parametrize("name,source", [("search", SEARCH)])
def test_on_the_host(tmp_path, name, source):
    src, exe = tmp_path / (name + ".cu"), tmp_path / name
    src.write_text(source)
    cmd = [_build._nvcc(), "-std=c++17", "-O1", "--expt-relaxed-constexpr", *_build.ARCH_FLAGS, "-I", _build.CSRC, "-I",
           _build.INCLUDE, "-o", str(exe), str(src)]
    built = subprocess.run(cmd, capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert ran.returncode == 0, ran.stdout


def test_searches_of_positions_take_the_safe_midpoint():
    """Adjacency and simplex positions go up to 2^31 - 2: no kernel that searches them adds two."""
    for name in ("links.cu", "simplices.cu"):
        text = open(os.path.join(_build.CSRC, name)).read()
        assert "midpoint(" in text or "lower_bound_i32(" in text
        assert "lo + hi" not in text and "lo[q] + hi[q]" not in text, name
