"""Loaded costs on the elimination hierarchy to the demand's fixed point: one pair
on a path 1/64 too long shows."""

import math

import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import dijkstra

from test_gpu_hierarchy import SHAPES, _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver

pytestmark = pytest.mark.gpu


def _shortest(net, dem):
    """Every positive pair's (trips, cost in whole 64ths); zones that are not passed
    through keep their outgoing links as origins only."""
    n, z = net.num_nodes, net.num_zones
    key = net.init * (n + 1) + net.term
    order = np.lexsort((net.fft, key))
    u = order[np.unique(key[order], return_index=True)[1]]
    through = net.init[u] >= net.first_thru_node
    trips, cost = [], []
    for o in range(1, z + 1):
        i0, i1 = dem.od_ptr[o], dem.od_ptr[o + 1]
        q, d = dem.od_demand[i0:i1], dem.od_dest[i0:i1]
        use = through | (net.init[u] == o)
        # (a stored zero is no link to scipy: 2^-30 a link is gone in the rounding)
        g = coo_matrix((net.fft[u][use] + 2.0 ** -30, (net.init[u][use], net.term[u][use])),
                       shape=(n + 1, n + 1)).tocsr()
        far = dijkstra(g, indices=o)[d]
        trips.append(q[d != o])
        cost.append(np.round(far[d != o] * 64.0) / 64.0)
    return np.concatenate(trips), np.concatenate(cost)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda c: "%dx%d" % (c["rows"], c["cols"]))
def test_loaded_cost(built_lib, shape):
    """Costs in whole 64ths, zero and equal ones among them, so whichever of several
    shortest paths is taken the loaded cost is exact: each pair's trips are rounded
    to 2^-s (half of that wrong at most), each link's volume to 53 bits."""
    c = dict(shape)
    S = c.pop("scen")
    net, dem = _net(seed=5, fft="integer", alpha=0.0, **c)
    with Solver(net, dem, precision="fp64") as s:
        _, on = _on_hierarchy(s, lambda: s.solve_scenarios(_scenarios(net, S, 6), max_iters=1))
        assert on
        x = s.flows_batch()[0]
    trips, cost = _shortest(net, dem)
    want = math.fsum(trips * cost)
    bits = min(40, 60 - math.ceil(math.log2(dem.od_demand.sum())))
    bound = 2.0 ** -(bits + 1) * cost.sum() + 2.0 ** -51 * want
    assert bound < trips.mean() / 64.0 / 100.0
    for row in (0, S // 2, S - 1):
        assert abs(math.fsum(x[row] * net.fft) - want) <= bound
