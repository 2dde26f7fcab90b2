"""The elimination-hierarchy path kernels (hier_kernels.cu) against the
label-correction kernels and against exact path costs, at the sizes where they
are chosen.  Networks: not square, groups of origins and tiles with
remainders, parallel links, self loops, centroids, zero costs."""

import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import dijkstra

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300._capi import TapGpuError
from traffic_assignment_gb300.synth import Demand, Network, Scenario, make_workload

pytestmark = pytest.mark.gpu


def _net(rows, cols, zones, seed, centroids=False, tree=False, fft="lognormal", alpha=0.15):
    """Two-way grid (or a spanning comb with a few cross streets), long links,
    parallel links and self loops; random zone nodes."""
    rng = np.random.default_rng(seed)
    i = np.arange(rows * cols).reshape(rows, cols)
    n = rows * cols
    across = np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)
    down = np.stack([i[:-1].ravel(), i[1:].ravel()], 1)
    if tree:
        keep = (down[:, 0] % cols == 0) | (rng.random(len(down)) < 0.08)
        down = down[keep]
    e = np.concatenate([across, down, rng.integers(0, n, (n // 60, 2))])
    e = e[e[:, 0] != e[:, 1]]
    u, v = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    again = rng.choice(len(u), len(u) // 30, replace=False)  # parallel links
    loops = rng.choice(n, 5, replace=False)
    u, v = np.concatenate([u, u[again], loops]), np.concatenate([v, v[again], loops])
    number = rng.permutation(n) + 1
    first = 1
    init, term = number[u], number[v]
    if centroids:  # zones 1..zones hang on street nodes by connectors
        first = zones + 1
        at = zones + rng.choice(n, zones, replace=False) + 1
        z = np.arange(1, zones + 1)
        init, term = np.concatenate([init + zones, z, at]), np.concatenate([term + zones, at, z])
        n += zones
    m = len(init)
    cost = (rng.integers(0, 400, m) / 64.0 if fft == "integer" else
            rng.lognormal(0.3, 0.6, m))
    order = np.lexsort((term, init))
    net = Network(num_nodes=n, num_zones=zones, first_thru_node=first, init=init[order],
                  term=term[order], capacity=rng.uniform(1500.0, 4000.0, m), length=np.ones(m),
                  fft=cost, alpha=np.full(m, alpha), beta=np.full(m, 4.0), speed=np.zeros(m),
                  toll=np.zeros(m), link_type=np.ones(m, np.int16))
    t = np.where(rng.random((zones, zones)) < 0.7, rng.uniform(0.0, 60.0, (zones, zones)), 0.0)
    o, d = np.nonzero(t)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(o + 1, minlength=zones + 1))])
    return net, Demand(num_zones=zones, od_ptr=ptr.astype(np.int64),
                       od_dest=(d + 1).astype(np.int64), od_demand=t[o, d])


def _scenarios(net, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for s in range(count):
        links = np.sort(rng.choice(net.num_links, 1 + s % 20, replace=False)).astype(np.int64)
        out.append(Scenario(f"s{s}", links, net.capacity[links] * rng.uniform(0.5, 2.0, len(links))))
    return out


def _on_hierarchy(s, run):
    """run() with the label-correction kernels' task counter: none ran."""
    s.set_timing(True)
    out = run()
    tasks = s.timing()["sssp_tasks"]
    s.set_timing(False)
    return out, tasks == 0


# (rows, cols, zones, scenarios): just above the small networks, remainders of
# the groups of 32 origins, a near-tree, several chunks of 32 columns
SHAPES = [
    dict(rows=23, cols=52, zones=97, scen=64),
    dict(rows=31, cols=77, zones=64, scen=96, tree=True),
    dict(rows=43, cols=83, zones=161, scen=96, centroids=True),
    dict(rows=70, cols=71, zones=333, scen=48),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda c: "%dx%d" % (c["rows"], c["cols"]))
def test_equals_label_correction_fp64(built_lib, shape):
    """The same trees, so the same flows: FP64 path costs differ by 2^-54 of
    the largest label between the two, far below any gap between two paths of
    random costs."""
    c = dict(shape)
    S = c.pop("scen")
    net, dem = _net(seed=3, **c)
    scen = _scenarios(net, S, 4)
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            r, on = _on_hierarchy(s, lambda: s.solve_scenarios(scen, max_iters=4))
            assert on == (variant == "default")
            out.append((s.flows_batch(), [x["total_cost"] for x in r], [x["relgap"] for x in r]))
    np.testing.assert_array_equal(out[0][0][0], out[1][0][0])
    np.testing.assert_array_equal(out[0][0][1], out[1][0][1])
    assert out[0][1:] == out[1][1:]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda c: "%dx%d" % (c["rows"], c["cols"]))
def test_exact_path_costs(built_lib, shape):
    """Fixed costs in whole 64ths, zero and equal ones among them: integer
    labels hold every path cost exactly, so whichever of several shortest
    paths is taken, the loaded cost is that of the shortest paths and the flow
    is conserved, to the fixed point of the demand (2^-40 of a trip)."""
    rtol = 1e-9
    c = dict(shape)
    S = c.pop("scen")
    net, dem = _net(seed=5, fft="integer", alpha=0.0, **c)
    with Solver(net, dem, precision="fp64") as s:
        _, on = _on_hierarchy(s, lambda: s.solve_scenarios(_scenarios(net, S, 6), max_iters=1))
        assert on
        x = s.flows_batch()[0]
    n, z = net.num_nodes, net.num_zones
    # shortest costs: the least of parallel links; links into zones that are not
    # passed through are kept only towards destinations
    key = net.init * (n + 1) + net.term
    order = np.lexsort((net.fft, key))
    u = order[np.unique(key[order], return_index=True)[1]]
    out = net.init[u] >= net.first_thru_node
    eps = 1e-12  # (a stored zero is no link to scipy)
    want = 0.0
    loads = np.zeros(n + 1)
    for o in range(1, z + 1):
        i0, i1 = dem.od_ptr[o], dem.od_ptr[o + 1]
        q, d = dem.od_demand[i0:i1].copy(), dem.od_dest[i0:i1]
        q[d == o] = 0.0
        use = out | (net.init[u] == o)
        g = coo_matrix((net.fft[u][use] + eps, (net.init[u][use], net.term[u][use])),
                       shape=(n + 1, n + 1)).tocsr()
        want += (dijkstra(g, indices=o)[d] * q).sum()
        loads[o] -= q.sum()
        np.add.at(loads, d, q)
    for s_ in (0, S // 2, S - 1):
        assert abs((x[s_] * net.fft).sum() - want) <= (rtol + 1e-7) * want
        net_in = np.bincount(net.term, x[s_], n + 1) - np.bincount(net.init, x[s_], n + 1)
        assert np.abs(net_in - loads).max() <= rtol * np.abs(dem.od_demand).sum()


@pytest.mark.parametrize("factor", [20.0, 100.0])
def test_labels_leave_the_integer_range(built_lib, factor):
    """A restart whose costs are 2^14 or 2^24 times the free-flow ones: the
    iteration is repeated at smaller exponents, or handed to the
    label-correction kernels."""
    net, dem = _net(43, 83, 161, seed=7)
    scen = _scenarios(net, 96, 8)
    x0 = factor * net.capacity
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            r = s.solve_scenarios(scen, max_iters=2, x0=x0)
            out.append((s.flows_batch()[0], [(x["total_cost"], x["objective"], x["iterations"]) for x in r]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]


def test_no_path_is_reported(built_lib):
    net, dem = _net(43, 83, 161, seed=9)
    cut = (net.term != 3) | (net.init == 3)  # zone 3 cannot be reached
    names = ("init", "term", "capacity", "length", "fft", "alpha", "beta", "speed", "toll", "link_type")
    net = Network(num_nodes=net.num_nodes, num_zones=net.num_zones,
                  first_thru_node=net.first_thru_node, **{k: getattr(net, k)[cut] for k in names})
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, sssp_variant=variant) as s:
            with pytest.raises(TapGpuError, match="no path"):
                s.solve_scenarios(_scenarios(net, 96, 1), max_iters=2)


def test_scenarios_own_links_and_demand(built_lib):
    """Absent links, changed parameters and trips by scenario: the flows of the
    label-correction kernels."""
    net, dem = _net(23, 52, 97, seed=11)
    S = 64
    rng = np.random.default_rng(12)
    edits, absent = [], []
    for s_ in range(S):
        k = np.sort(rng.choice(net.num_links, 4, replace=False))
        edits.append((k, net.fft[k] * 1.5, net.alpha[k], net.beta[k]))
        # one of two parallel links: the network stays connected
        pair = np.nonzero((net.init[1:] == net.init[:-1]) & (net.term[1:] == net.term[:-1]))[0]
        absent.append(np.sort(rng.choice(pair, 3, replace=False)))
    trips = dem.od_demand[None] * rng.choice([0.0, 0.5, 1.0, 1.5], (S, 1))
    trips[:, ::7] = 0.0
    trips[0] = dem.od_demand
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            s.set_scenario_links(edits, absent)
            s.set_scenario_demand(trips)
            r, on = _on_hierarchy(s, lambda: s.solve_scenarios(_scenarios(net, S, 13), max_iters=3))
            assert on == (variant == "default")
            out.append((s.flows_batch()[0], np.array([x["total_cost"] for x in r])))
    for s_ in range(S):
        assert (out[0][0][s_][absent[s_]] == 0).all()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def test_paths_change_with_the_batch(built_lib):
    """One context solves one scenario (label correction), many (hierarchy) and
    one again, and advances batches stepwise: the same bits each time."""
    net, dem = _net(43, 83, 161, seed=15)
    scen = _scenarios(net, 96, 16)
    with Solver(net, dem, precision="fp64") as s:
        s.solve(max_iters=3)
        one = s.flows()[0]
        s.solve_scenarios(scen, max_iters=5)
        many = s.flows_batch()[0]
        s.solve(max_iters=3)
        np.testing.assert_array_equal(one, s.flows()[0])
        s.solve_scenarios(scen, max_iters=2)
        s.run_iterations(3)
        np.testing.assert_array_equal(many, s.flows_batch()[0])


def test_one_loading_at_given_costs(built_lib):
    """aon() of a context whose single loadings pay, at the free-flow costs'
    scale, far from it (the exponent is found anew) and in between solves: the
    label-correction kernels' volumes."""
    net, dem = make_workload("grid10k")
    rng = np.random.default_rng(17)
    w = net.fft * rng.lognormal(0.0, 0.5, net.num_links)
    out = []
    for variant in ("default", "nearfar_queue"):
        with Solver(net, dem, precision="fp64", sssp_variant=variant) as s:
            y, on = _on_hierarchy(s, lambda: [s.aon(w * f) for f in (1.0, 2.0 ** 12, 2.0 ** -30)])
            assert on == (variant == "default")
            y.append(s.aon(w * 2.0 ** 40))  # (beyond the exponents that are tried)
            s.solve(max_iters=2)
            y += [s.aon(w), s.flows()[0]]
            out.append(y)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    for y in out[0][1:4]:  # a power of two changes no path
        np.testing.assert_array_equal(y, out[0][0])
