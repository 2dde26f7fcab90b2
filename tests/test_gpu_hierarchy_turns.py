"""Scenarios that take turns in the elimination hierarchy's buffers while some of
them leave the integer labels' range: every scenario's flows are its own."""

import numpy as np
import pytest

from test_gpu_hierarchy import _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300._capi import TapGpuError

pytestmark = pytest.mark.gpu


# one slot for all; a few (a scenario's buffers take 15 to 20 MB); all at once
@pytest.mark.parametrize("limit", [1, 100 << 20, 500 << 20, 0])
def test_own_flows(built_lib, limit):
    """Trips of a third of the scenarios are 12 to 80 times the base's (their first
    costs are 2^14 to 2^25 times the free-flow ones, and fall again), of others
    as they are or next to nothing: some scenarios pause for a larger range, some
    for a finer unit, their neighbours not.  (Sums over links, as the excess, are
    added up by as many blocks as the launch's scenarios leave, so their last bit
    depends on who paused; flows, costs and steps do not.)"""
    net, dem = _net(43, 83, 161, seed=21)
    S = 96
    scen = _scenarios(net, S, 22)
    rng = np.random.default_rng(23)
    factor = np.where(np.arange(S) % 3 == 0, rng.uniform(12.0, 80.0, S),
                      rng.choice([0.01, 0.7, 1.0], S))
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            if variant == "default":
                s.set_hierarchy_limit(limit)
            s.set_scenario_demand(dem.od_demand[None] * factor[:, None])
            r = s.solve_scenarios(scen, max_iters=6)
            x, t = s.flows_batch()
            out.append((x, t, [(v["iterations"], v["lambda_last"]) for v in r]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


def test_turns_without_pauses(built_lib):
    net, dem = _net(43, 83, 161, seed=25)
    scen = _scenarios(net, 40, 26)
    out = []
    for limit in (0, 1):
        with Solver(net, dem, precision="fp64") as s:
            s.set_hierarchy_limit(limit)
            _, on = _on_hierarchy(s, lambda: s.solve_scenarios(scen, max_iters=3))
            assert on
            s.set_hierarchy_limit(limit)  # (gives the buffers back between two calls)
            with pytest.raises(TapGpuError):
                s.run_iterations(1)
            s.solve_scenarios(scen, max_iters=3)
            out.append(s.flows_batch()[0])
    np.testing.assert_array_equal(out[0], out[1])
