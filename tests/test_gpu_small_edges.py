"""The small networks' shortest paths with their edges in registers, at the
edges of its dispatch (whole and ragged edges per thread), against the
label-correction rounds: the same labels, so the same bits."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Demand, Network

pytestmark = pytest.mark.gpu


def _net(nodes, links, first_thru, seed):
    """A ring through all thru nodes, zones tied to it both ways, random links;
    link count exact, parallel links and self loops among them."""
    rng = np.random.default_rng(seed)
    z = first_thru - 1 if first_thru > 1 else min(3, nodes)
    thru = np.arange(first_thru, nodes + 1)
    u, v = [thru], [np.roll(thru, -1)]
    if first_thru > 1:
        at = rng.choice(thru, z)
        u += [np.arange(1, z + 1), at]
        v += [at, np.arange(1, z + 1)]
    u, v = np.concatenate(u), np.concatenate(v)
    more = links - len(u)
    assert more >= 0
    u = np.concatenate([u, rng.choice(thru, more)])
    v = np.concatenate([v, rng.choice(thru, more)])
    net = Network(num_nodes=nodes, num_zones=z, first_thru_node=first_thru, init=u, term=v,
                  capacity=np.full(links, 1e3), length=np.ones(links),
                  fft=rng.lognormal(0.0, 0.7, links) * (rng.random(links) > 0.02),
                  alpha=np.full(links, 0.15), beta=np.full(links, 4.0), speed=np.zeros(links),
                  toll=np.zeros(links), link_type=np.ones(links, np.int16))
    o, d = np.divmod(np.arange(z * z), z)
    dem = Demand(num_zones=z, od_ptr=np.concatenate([[0], np.arange(z + 1) * z]).astype(np.int64),
                 od_dest=(d + 1).astype(np.int64), od_demand=rng.uniform(0.0, 50.0, z * z) * (o != d))
    return net, dem


@pytest.mark.parametrize("nodes,links,first_thru", [
    (2, 2, 1), (5, 31, 1), (200, 511, 1), (301, 512, 1), (420, 513, 41), (700, 1024, 1),
    (900, 1537, 88), (1300, 2049, 1), (1900, 3000, 60), (2400, 3584, 1), (4095, 4096, 1)])
def test_equals_rounds(built_lib, nodes, links, first_thru):
    net, dem = _net(nodes, links, first_thru, nodes)
    rng = np.random.default_rng(1)
    w = net.fft * rng.uniform(0.5, 2.0, links)
    src = np.unique(np.concatenate([[1, nodes], rng.integers(1, nodes + 1, 9)]))
    out = {}
    for precision in ("fp64", "fp32"):
        for variant in ("small", "rounds"):
            # (rounds by name: the small kernel is the library's choice here)
            kw = {} if variant == "small" else dict(sssp_variant="rounds")
            with Solver(net, dem if nodes > 2 else None, precision=precision, **kw) as s:
                dist = s.sssp(w, src, want_pred=False)[0]
                vol = None
                if nodes > 2:
                    s.solve(max_iters=3)
                    vol = np.concatenate([s.aon(w), s.flows()[0]])
                out[precision, variant] = dist, vol
        np.testing.assert_array_equal(out[precision, "small"][0], out[precision, "rounds"][0])
        if nodes > 2:
            np.testing.assert_array_equal(out[precision, "small"][1], out[precision, "rounds"][1])
