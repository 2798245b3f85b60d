"""The most views of one half-turn angle within a range of table positions
(bp_most_views): the searches of an ordered table against the walk over all views,
for rising, falling, standing, stepped and unordered tables, whole and broken half
turns, ranges that hold none, some and all views, and bounds on a position."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "wfbp_internal.h"
#include <stdio.h>
#include <random>
int main() {
  std::mt19937 rng(5);
  auto uni = [&](double a, double b) { return (float)std::uniform_real_distribution<double>(a, b)(rng); };
  long n = 0, bad = 0, ordered = 0;
  for (int P2 : {1, 2, 7, 48, 205})
    for (int K : {1, 2, 5, 13})
      for (int kind = 0; kind < 6; kind++) {
        std::vector<float> t((size_t)P2 * K + 3);
        float z = uni(-100, 100);
        for (auto& v : t) {
          if (kind == 0) z += uni(0.01, 1);
          if (kind == 1) z -= uni(0.01, 1);
          if (kind == 3 && rng() % 5 == 0) z += 1;
          if (kind == 4 && rng() % 5 == 0) z -= 1;
          if (kind == 5) z += uni(-1, 1);
          v = z;
        }
        const int order = bp_table_order(t.data(), P2 * K);
        ordered += order != 0;
        for (int i = 0; i < 200; i++) {
          const float a = i % 3 ? t[rng() % t.size()] : uni(-300, 300), b = i % 2 ? t[rng() % t.size()] : uni(-300, 300);
          const float lo = a < b ? a : b, hi = a < b ? b : a;
          n++;
          bad += bp_most_views(t.data(), order, P2, K, lo, hi) != bp_most_views(t.data(), 0, P2, K, lo, hi);
        }
      }
  printf("%ld %ld %ld\n", n, ordered, bad);
  return 0;
}
"""


def test_searches_equal_the_walk(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    from freect_b200 import build_lib
    cuda = os.path.join(os.path.dirname(os.path.dirname(build_lib.nvcc())), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + cuda, "-I" + os.path.join(ROOT, "freect_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    n, ordered, bad = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n == 24000 and ordered >= 100 and bad == 0
