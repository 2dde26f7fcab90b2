"""Step sizes with a known answer: two equal routes, started a little off their
equilibrium, so that the best step is 1.5 x 2^-k (tap/tap_functions.c:469-507
takes 2^-k)."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Demand, Network

pytestmark = pytest.mark.gpu

D = 1024.0


def _net(spare):
    """Two parallel links 1 -> 2, one back, and `spare` links that carry nothing."""
    n = 2 + spare + 1
    u = np.concatenate([[1, 1, 2], np.arange(3, 3 + spare)])
    v = np.concatenate([[2, 2, 1], np.arange(4, 4 + spare)])
    m = len(u)
    return Network(num_nodes=n, num_zones=2, first_thru_node=1, init=u, term=v,
                   capacity=np.full(m, 600.0), length=np.ones(m), fft=np.full(m, 3.0),
                   alpha=np.full(m, 0.15), beta=np.full(m, 4.0), speed=np.zeros(m), toll=np.zeros(m),
                   link_type=np.ones(m, np.int16)), Demand(
                       num_zones=2, od_ptr=np.array([0, 0, 1, 1]), od_dest=np.array([2]),
                       od_demand=np.array([D]))


# one launch for the whole tail; 64-thread blocks; 256-thread blocks
@pytest.mark.parametrize("spare", [0, 2500, 6000, 45000])
@pytest.mark.parametrize("rule", ["reference", "exact"])
def test_known_steps(built_lib, spare, rule):
    net, dem = _net(spare)
    # first and last candidates of the passes, and beyond those of the grid
    for k in (1, 2, 11, 12, 13, 23, 24, 25, 26, 30):
        best = 1.5 * 2.0 ** -k if k > 1 else 0.75
        # x1 = D/2 + e, d1 = -x1: level again at the step e / (D/2 + e)
        e = best * (D / 2) / (1.0 - best)
        x0 = np.zeros(net.num_links)
        x0[:2] = D / 2 + e, D / 2 - e
        with Solver(net, dem, precision="fp64", line_search=rule) as s:
            r = s.solve(max_iters=1, x0=x0)
            assert r["error_bits"] == 0
            x, _ = s.flows()
        if rule == "reference":
            assert r["lambda_last"] == 2.0 ** -k
        else:
            # costs are rounded to 2^-53 of their own: a step to about 2^-52
            assert abs(r["lambda_last"] - best) <= 2.0 ** -49
        np.testing.assert_allclose(x[:2].sum(), D, rtol=1e-12)
