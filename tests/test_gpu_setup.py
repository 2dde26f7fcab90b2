"""Contexts that may take the elimination hierarchy: set up without waiting for its
plan, which the first solve or loading asks for."""

import os
import signal
import time

import numpy as np
import pytest

from test_gpu_hierarchy import _net, _on_hierarchy
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300._capi import TapGpuError
from traffic_assignment_gb300.synth import make_workload

pytestmark = pytest.mark.gpu


def _shortest(make, count=6):
    best = 1e9
    for _ in range(count):
        t0 = time.perf_counter()
        s = make()
        best = min(best, time.perf_counter() - t0)
        s.close()
    return best


@pytest.mark.parametrize("with_demand", [True, False])
def test_setup_does_not_wait(built_lib, with_demand):
    """40,000 nodes: 7 ms without a plan, 41 ms where the setup waited for it."""
    net, dem = _net(200, 200, 150, seed=61)
    if not with_demand:
        dem = None
    plain = _shortest(lambda: Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue"))
    assert _shortest(lambda: Solver(net, dem, precision="fp64")) <= 2.0 * plain + 3e-3


def test_first_uses(built_lib):
    """Closed at once; a loading, a solve, or trees and then a solve first: the
    hierarchy and label correction's results."""
    net, dem = make_workload("grid10k")
    w = net.fft * np.random.default_rng(62).lognormal(0.0, 0.5, net.num_links)
    with Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue") as s:
        y = s.aon(w)
        dist, _ = s.sssp(w, [1, 77])
        s.solve(max_iters=2)
        x = s.flows()[0]
    for _ in range(3):
        Solver(net, dem, precision="fp64").close()
    with Solver(net, dem, precision="fp64") as s:
        with pytest.raises(TapGpuError):
            s.run_iterations(1)
        got, on = _on_hierarchy(s, lambda: s.aon(w))
        assert on
        np.testing.assert_array_equal(got, y)
    with Solver(net, dem, precision="fp64") as s:
        _, on = _on_hierarchy(s, lambda: s.solve(max_iters=2))
        assert on
        np.testing.assert_array_equal(s.flows()[0], x)
    with Solver(net, dem, precision="fp64") as s:
        np.testing.assert_array_equal(s.sssp(w, [1, 77])[0], dist)
        _, on = _on_hierarchy(s, lambda: s.solve(max_iters=2))
        assert on
        np.testing.assert_array_equal(s.flows()[0], x)


def _threads():
    return set(os.listdir("/proc/self/task"))


def test_signals_are_the_callers(built_lib):
    """The plan's thread goes on after the setup, perhaps while the caller blocks
    signals in its own threads to wait for them: none may be delivered to it."""
    net, dem = _net(200, 200, 150, seed=63)
    Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue").close()
    blocked = []
    for _ in range(3):
        before = _threads()
        with Solver(net, dem, precision="fp64"):
            for t in _threads() - before:
                try:
                    with open(f"/proc/self/task/{t}/status") as f:
                        mask = int(next(x for x in f if x.startswith("SigBlk")).split()[1], 16)
                except (OSError, StopIteration):
                    continue  # (it has ended)
                blocked += [bool(mask >> (n - 1) & 1) for n in
                            (signal.SIGINT, signal.SIGTERM, signal.SIGUSR1, signal.SIGUSR2)]
    assert blocked and all(blocked)
