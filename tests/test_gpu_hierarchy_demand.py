"""Few pairs of many zones: demand scenarios are accepted and solved whether or not
the hierarchy's table of all pairs of zones fits."""

import numpy as np
import pytest

from test_gpu_hierarchy import _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Demand

pytestmark = pytest.mark.gpu


def _sparse(rows, cols, zones, seed):
    net, _ = _net(rows, cols, zones, seed)
    rng = np.random.default_rng(seed + 1)
    o = np.sort(np.concatenate([np.arange(1, zones + 1), rng.integers(1, zones + 1, zones // 5)]))
    d = rng.integers(1, zones + 1, len(o))
    d[: zones] = np.where(d[: zones] == o[: zones], 1 + o[: zones] % zones, d[: zones])
    ptr = np.concatenate([[0], np.cumsum(np.bincount(o, minlength=zones + 1))])
    return net, Demand(num_zones=zones, od_ptr=ptr.astype(np.int64), od_dest=d.astype(np.int64),
                       od_demand=rng.uniform(1.0, 60.0, len(o)))


def test_tables_that_do_not_fit(built_lib):
    """5,000 zones, 6,000 pairs: about 130 MB of table (3,500 destinations) a
    scenario, 700 GB for 5,500 of them, 26 GiB for 210."""
    net, dem = _sparse(70, 72, 5000, 41)
    rng = np.random.default_rng(43)
    with Solver(net, dem, precision="fp64") as s:
        s.set_scenario_demand(np.tile(dem.od_demand, (5500, 1)))
        s.set_scenario_demand(None)
        trips = dem.od_demand[None] * rng.uniform(0.5, 1.5, (210, 1))
        s.set_scenario_demand(trips)
        _, on = _on_hierarchy(s, lambda: s.solve_scenarios(_scenarios(net, 210, 44), max_iters=1))
        assert not on
        x = s.flows_batch()[0]
        s.set_scenario_demand(trips[:8])  # (a table that fits)
        s.solve_scenarios(_scenarios(net, 8, 44), max_iters=1)
        np.testing.assert_array_equal(s.flows_batch()[0], x[:8])
        s.set_scenario_demand(None)
        _, on = _on_hierarchy(s, lambda: s.solve(max_iters=1))
        assert on
        one = s.flows()[0]
    with Solver(net, dem, precision="fp64", sssp_variant="nearfar_queue") as s:
        s.solve(max_iters=1)
        np.testing.assert_array_equal(one, s.flows()[0])


def test_base_demand_in_a_new_unit(built_lib):
    """Demand scenarios with more trips lower the fixed point's unit: the base
    demand's table is made again, before and after its first use."""
    net, dem = _sparse(70, 72, 300, 45)
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            got = []
            for factor in (1.0, 2.0 ** 9, 2.0 ** 14):
                if factor > 1.0:
                    s.set_scenario_demand(np.tile(dem.od_demand * factor, (64, 1)))
                    s.solve_scenarios(_scenarios(net, 64, 46), max_iters=2)
                    got.append(s.flows_batch()[0])
                    s.set_scenario_demand(None)
                s.solve_scenarios(_scenarios(net, 64, 46), max_iters=2)
                got.append(s.flows_batch()[0])
            out.append(got)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
