"""The elimination hierarchy on networks with hubs, which its order puts last,
against label correction."""

import numpy as np
import pytest

from test_gpu_hierarchy import _net, _on_hierarchy, _scenarios
from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Network

pytestmark = pytest.mark.gpu


def _with_hubs(net, leaves, hubs, seed):
    """Links to and from each hub node for `leaves` street nodes, about as dear as
    ten street links."""
    rng = np.random.default_rng(seed)
    streets = np.arange(net.first_thru_node, net.num_nodes + 1)
    u, v = [net.init], [net.term]
    for h in hubs:
        at = rng.choice(np.setdiff1d(streets, hubs), leaves, replace=False)
        u += [np.full(leaves, h), at]
        v += [at, np.full(leaves, h)]
    u, v = np.concatenate(u), np.concatenate(v)
    m, old = len(u), net.num_links
    fft = np.concatenate([net.fft, rng.lognormal(2.2, 0.6, m - old)])
    cap = np.concatenate([net.capacity, rng.uniform(1500.0, 4000.0, m - old)])
    order = np.lexsort((v, u))
    return Network(num_nodes=max(net.num_nodes, max(hubs)), num_zones=net.num_zones,
                   first_thru_node=net.first_thru_node, init=u[order], term=v[order],
                   capacity=cap[order], length=np.ones(m), fft=fft[order], alpha=np.full(m, 0.15),
                   beta=np.full(m, 4.0), speed=np.zeros(m), toll=np.zeros(m),
                   link_type=np.ones(m, np.int16))


@pytest.mark.parametrize("centroids", [False, True])
def test_equals_label_correction(built_lib, centroids):
    """1,200 leaves each, 10 sqrt(n) is 770: two hubs that are new nodes and one
    that is a zone (without centroids)."""
    net, dem = _net(70, 84, 161, seed=51, centroids=centroids)
    hubs = [net.num_nodes + 1, net.num_nodes + 2] + ([] if centroids else [5])
    net = _with_hubs(net, 1200, hubs, 52)
    scen = _scenarios(net, 64, 53)
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            r, on = _on_hierarchy(s, lambda: s.solve_scenarios(scen, max_iters=4))
            assert on == (variant == "default")
            out.append((s.flows_batch(), [x["total_cost"] for x in r]))
    np.testing.assert_array_equal(out[0][0][0], out[1][0][0])
    np.testing.assert_array_equal(out[0][0][1], out[1][0][1])
    assert out[0][1] == out[1][1]
