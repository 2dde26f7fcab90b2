"""Calls after one that found no device memory: refused again, or solved, but never
run on arrays that are not there."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300._capi import TapGpuError
from traffic_assignment_gb300.synth import Scenario, make_small24

pytestmark = pytest.mark.gpu


def _plain(net, count):
    return [Scenario(f"s{i}", np.zeros(0, np.int64), np.zeros(0)) for i in range(count)]


def test_tape_that_does_not_fit(built_lib):
    """Directions of 512 scenarios x 2,000,000 iterations x 76 links: 622 GB, asked
    for after the other arrays of the scenarios are there."""
    net, dem = make_small24()
    with Solver(net, dem) as s:
        want = s.solve(max_iters=5), s.flows()[0]
    with Solver(net, dem, record_tape=True, tape_capacity=2_000_000) as s:
        for count in (512, 512, 500):
            with pytest.raises(TapGpuError, match="cudaMalloc"):
                s.solve_scenarios(_plain(net, count), max_iters=5)
            for later in (lambda: s.run_iterations(1), lambda: s.advance(1), s.flows):
                with pytest.raises(TapGpuError):
                    later()
        s.set_capacity(net.capacity)
        got = s.solve(max_iters=5), s.flows()[0]
        assert got[0] == want[0]
        np.testing.assert_array_equal(got[1], want[1])
        s.solve_scenarios(_plain(net, 1), max_iters=5)
        np.testing.assert_array_equal(s.flows()[0], want[1])
