"""Rows that the shortest-path API widens at once, up to the largest node count."""

import os
import shutil
import subprocess

import pytest


def test_rows_at_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc absent")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    # (rows, nodes): small, 64 MiB exactly, and where 8 n wraps to negative and to zero
    cases = [(5, 25), (10000, 1 << 13), (300, 100001), (7, (1 << 28) - 1), (7, 1 << 28),
             (7, (1 << 28) + 1), (7, 1 << 29), (7, (1 << 30) + 1)]
    src = tmp_path / "rows.cu"
    calls = "".join(f'std::printf("%lld ", static_cast<long long>(tapgpu::rows_at_once({r}, {n})));'
                    for r, n in cases)
    src.write_text('#include <cstdio>\n#include "solver.cuh"\nint main() { ' + calls + " return 0; }\n")
    exe = tmp_path / "rows"
    subprocess.run([nvcc, "-std=c++17", "-I", os.path.join(root, "include"), "-I",
                    os.path.join(root, "traffic_assignment_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    got = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in got] == [max(1, min(r, (64 << 20) // (8 * n))) for r, n in cases]
