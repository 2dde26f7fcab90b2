"""The elimination hierarchy's host plan of networks with hubs: made in time that
grows with the links, not with the square of a hub's."""

import os
import shutil
import subprocess

import pytest

MAIN = r"""
#include <chrono>
#include <cstdio>
#include "hierarchy.h"
int main() {
  for (int hubs : {1, 3}) {
    const int n = 100000;
    std::vector<int> u, v;
    for (int i = hubs + 1; i < n; ++i)
      for (int h = 1; h <= hubs; ++h) {
        u.push_back(i); v.push_back(h);
        u.push_back(h); v.push_back(i);
      }
    std::vector<char> dests(n, 1);
    tapgpu::HierPlan p;
    const auto t0 = std::chrono::steady_clock::now();
    const bool ok = tapgpu::hier_build(n, static_cast<int>(u.size()), u.data(), v.data(), 1, dests,
                                       80.0 * n, 1e11, p);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    int above = 0;  // positions of the hubs among the last ones
    for (int h = 1; ok && h <= hubs; ++h) above += p.pos[h] >= n - 1 - hubs;
    std::printf("%d %d %f\n", ok, above, s);
  }
}
"""


def test_hubs(tmp_path):
    """Stars of 100,000 leaves around one hub and around three: 0.04 and 0.06 s (with
    every leaf going through its hubs' neighbours 5.6 and 5.5 s), hubs on top."""
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ absent")
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "traffic_assignment_gb300", "csrc")
    src, exe = tmp_path / "hubs.cpp", tmp_path / "hubs"
    src.write_text(MAIN)
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", csrc, str(src), os.path.join(csrc, "hierarchy.cpp"),
                    "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for hubs, line in zip((1, 3), out):
        ok, above, seconds = line.split()
        assert int(ok) == 1 and int(above) == hubs
        assert float(seconds) < 1.5
