"""profile_iteration on the elimination hierarchy when labels leave the integers'
range: the iterations it reports were made, and the solve goes on from them."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import make_workload

pytestmark = pytest.mark.gpu


def test_paused_iterations_are_repeated(built_lib):
    net, dem = make_workload("grid10k")
    x0 = 20.0 * net.capacity  # costs 2^14 times the free-flow ones
    with Solver(net, dem, precision="fp64") as s:
        s.begin(max_iters=50, x0=x0)
        ms = s.profile_iteration(3)
        assert all(v > 0 for v in ms.values())
        n = len(s.trace())
        assert n >= 3
        x = s.flows()[0]
        s.solve(max_iters=2)
        after = s.flows()[0]
    with Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue") as s:
        s.solve(max_iters=n, x0=x0)
        np.testing.assert_array_equal(x, s.flows()[0])
        s.solve(max_iters=2)
        np.testing.assert_array_equal(after, s.flows()[0])
