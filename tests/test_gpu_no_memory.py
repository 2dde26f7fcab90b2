"""Calls after one that found no device memory: refused again, or solved, but never
run on arrays that are not there."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300._capi import TapGpuError
from traffic_assignment_gb300.synth import Demand, Network, Scenario, make_small24

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


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_path_records_that_do_not_fit(built_lib, precision):
    """Padded records of 12,000 scenarios x 800,001 nodes: 307 GB (FP32; FP64 twice
    that), asked for after the first records of 24 links each are there."""
    n = 800_000
    u = np.r_[np.arange(1, 13), np.arange(2, 14)]
    v = np.r_[np.arange(2, 14), np.arange(1, 13)]
    m = len(u)
    net = Network(num_nodes=n, num_zones=13, first_thru_node=1, init=u, term=v,
                  capacity=np.full(m, 500.0), length=np.ones(m), fft=1.0 + np.arange(m) / 8.0,
                  alpha=np.full(m, 0.15), beta=np.full(m, 4.0), speed=np.zeros(m), toll=np.zeros(m),
                  link_type=np.ones(m, np.int16))
    dem = Demand(num_zones=13, od_ptr=np.r_[0, 0, np.full(13, 2)], od_dest=np.array([13, 5]),
                 od_demand=np.array([100.0, 50.0]))
    with Solver(net, dem, precision=precision, sssp_variant="nearfar_queue") as s:
        want = s.solve(max_iters=2), s.flows()[0]
        for _ in range(2):
            with pytest.raises(TapGpuError, match="cudaMalloc"):
                s.solve_scenarios(_plain(net, 12_000), max_iters=2)
            for later in (lambda: s.run_iterations(1), lambda: s.advance(1),
                          lambda: s.profile_iteration(1)):
                with pytest.raises(TapGpuError):
                    later()
        assert s.sssp(net.fft, [1])[0][0, 13] == net.fft[:12].sum()
        np.testing.assert_array_equal(s.aon(net.fft), want[1])
        again = s.solve(max_iters=2), s.flows()[0]
        assert again[0] == want[0]
        np.testing.assert_array_equal(again[1], want[1])
