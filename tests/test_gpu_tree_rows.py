"""tapgpu_sssp's results on the way to the caller's arrays: links in any order,
nodes out of reach, more predecessors than one block of the wide form holds."""

import numpy as np
import pytest

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Network

pytestmark = pytest.mark.gpu


def _net(rows, cols, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(1, rows * cols + 1).reshape(rows, cols)
    e = np.concatenate([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                        np.stack([i[:-1].ravel(), i[1:].ravel()], 1)])
    e = np.concatenate([e, e[:, ::-1]])
    e = e[e[:, 1] != rows * cols]  # the last node has no link to it
    e = e[rng.permutation(len(e))]  # links not sorted by node
    m = len(e)
    return Network(num_nodes=rows * cols, num_zones=4, first_thru_node=1, init=e[:, 0], term=e[:, 1],
                   capacity=np.full(m, 1e3), length=np.ones(m), fft=rng.lognormal(0.0, 0.5, m),
                   alpha=np.full(m, 0.15), beta=np.full(m, 4.0), speed=np.zeros(m), toll=np.zeros(m),
                   link_type=np.ones(m, np.int16))


# one row; whole blocks and a remainder (8 bytes x nodes x sources over 64 MiB)
@pytest.mark.parametrize("rows,cols,sources", [(5, 7, 1), (29, 31, 33), (90, 101, 1111)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_rows_are_trees(built_lib, rows, cols, sources, precision):
    net = _net(rows, cols, 3)
    n = net.num_nodes
    rng = np.random.default_rng(4)
    w = net.fft * rng.uniform(1.0, 2.0, net.num_links)
    src = rng.integers(1, n + 1, sources)
    src[-1] = 1
    with Solver(net, None, precision=precision) as s:
        first = s.sssp(w, src[-1:])  # (buffers for one row, then for all, then again one)
        dist, pred = s.sssp(w, src)
        last = s.sssp(w, src[-1:])
        only = s.sssp(w, src[:3], want_pred=False)[0]
    for d, p in (first, last):
        np.testing.assert_array_equal(d[0], dist[-1])
        np.testing.assert_array_equal(p[0], pred[-1])
    np.testing.assert_array_equal(only, dist[:3])
    assert dist.dtype == np.float64 and pred.dtype == np.int64
    big = np.finfo(np.float64).max
    row = np.arange(sources)
    # node 0 and the last node (unless it is the source) are out of reach
    out = np.zeros(dist.shape, bool)
    out[:, 0] = True
    out[:, n] = src != n
    np.testing.assert_array_equal(dist == big, out)
    assert (dist[row, src] == 0).all()
    none = out.copy()
    none[row, src] = True
    np.testing.assert_array_equal(pred == -1, none)
    # a predecessor leads to its node and its label, and no link does better
    r, v = np.nonzero(~none)
    k = pred[r, v]
    np.testing.assert_array_equal(net.term[k], v)
    np.testing.assert_array_equal(dist[r, net.init[k]] + w[k], dist[r, v])
    few = dist[:: max(1, sources // 40)]
    reach = few[:, net.init] < big
    assert (few[:, net.term][reach] <= (few[:, net.init] + w)[reach]).all()
