"""Costs spread over more of the integer labels' bits than ordinary links can be
told apart by: the label-correction kernels take those iterations."""

import numpy as np
import pytest

from test_gpu_hierarchy import _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import make_workload

pytestmark = pytest.mark.gpu


def _twins(net, rel):
    """Of every two parallel links the first is `rel` dearer than the second."""
    pair = np.nonzero((net.init[1:] == net.init[:-1]) & (net.term[1:] == net.term[:-1]))[0]
    net.fft[pair] = net.fft[pair + 1] * (1.0 + rel)
    return pair


@pytest.mark.parametrize("far", [0, 30, 40])
def test_near_ties_beside_a_far_zone(built_lib, far):
    """Every way into one zone costs 2^far times an ordinary link, twins differ by
    2^-18 of their cost: labels of 2^56 units for the far zone would leave an
    ordinary link about 2^(46 - far)."""
    net, dem = _net(43, 83, 161, seed=31)
    _twins(net, 2.0 ** -18)
    net.fft[(net.term == 7) & (net.init != 7)] *= 2.0 ** far
    scen = _scenarios(net, 96, 32)
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            r, on = _on_hierarchy(s, lambda: s.solve_scenarios(scen, max_iters=4))
            assert on == (variant == "default" and far == 0)
            x, t = s.flows_batch()
            s.run_iterations(2)
            out.append((x, t, s.flows_batch()[0], [v["lambda_last"] for v in r]))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_some_scenarios_spread(built_lib):
    """The far zone is far in every third scenario only, by its own link records."""
    net, dem = _net(43, 83, 161, seed=33)
    _twins(net, 2.0 ** -18)
    S = 96
    k = np.nonzero((net.term == 7) & (net.init != 7))[0]
    edits = [(k, net.fft[k] * 2.0 ** 40, net.alpha[k], net.beta[k]) if i % 3 == 0 else None
             for i in range(S)]
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            s.set_scenario_links(edits)
            s.solve_scenarios(_scenarios(net, S, 34), max_iters=5)
            out.append(s.flows_batch())
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def test_single_calls(built_lib):
    """aon, solve, begin / advance and profile_iteration of one scenario."""
    net, dem = make_workload("grid10k")
    k = np.nonzero(net.term == 7)[0]
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            w = net.fft.copy()
            got = [s.aon(w)]
            w[k] *= 2.0 ** 45
            got.append(s.aon(w))
            x0 = 0.5 * net.capacity
            x0[k] *= 2.0 ** 12
            s.solve(max_iters=5, x0=x0)
            got.append(s.flows()[0])
            s.begin(max_iters=9, x0=x0)
            while not s.advance(2)[0]:
                pass
            got += s.flows()
            s.begin(max_iters=9, x0=x0)
            s.profile_iteration(3)
            got.append(s.flows()[0] if len(s.trace()) >= 3 else None)
            n = len(s.trace())
        out.append((got, n))
    with Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue") as s:
        s.solve(max_iters=out[0][1], x0=x0)
        out[1][0][-1] = s.flows()[0]
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
