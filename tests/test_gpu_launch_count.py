"""The kernels that a context counts where the elimination hierarchy takes its
iterations and loadings."""

import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import make_workload

pytestmark = pytest.mark.gpu


def test_launches_are_counted(built_lib):
    """One loading's launches through aon(), and as part of an iteration, which has
    two line-search passes, their rest and the step besides."""
    net, dem = make_workload("grid10k")
    with Solver(net, dem, precision="fp64", use_graphs=False) as s:
        s.solve(max_iters=1)
        s.set_timing(True)
        s.run_iterations(3)
        iterations = s.timing()
        s.set_timing(True)
        s.aon(net.fft)
        loading = s.timing()
    assert iterations["sssp_tasks"] == 0 and loading["sssp_tasks"] == 0
    assert loading["kernel_launches"] > 25
    assert iterations["kernel_launches"] == 3 * (loading["kernel_launches"] + 4)
