"""The autotuner where the library's own choice is the elimination hierarchy, which
no explicit launch shape reaches."""

import pytest

from test_gpu_hierarchy import _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300 import autotune as A

pytestmark = pytest.mark.gpu


def test_the_librarys_choice_is_a_candidate(built_lib):
    """3,569 nodes, 161 zones, 64 FP64 scenarios: paths and loading take about half
    as long on the hierarchy as with any label-correction shape."""
    net, dem = _net(43, 83, 161, seed=71)
    scen = _scenarios(net, 64, 72)
    r = A.tune(net, dem, "fp64", iters=2, warm_iters=5, quick=True, scenario_list=scen)
    assert r.best.sssp_variant == "default"
    with Solver(net, dem, precision="fp64", **r.solver_kwargs(net)) as s:
        _, on = _on_hierarchy(s, lambda: s.solve_scenarios(scen, max_iters=2))
        assert on
