"""What this framework is measured on: calls of its public entry points over the
range of networks, precisions and modes that it is used with.

Every input (network, demand, upgrade scenarios, warm start) is generated here
from the seed alone, with the shapes and value distributions of the
repository's own workloads (the 24-, 416-, 454-, 3,600-, 10,000- and
100,000-node networks of its tests and benchmark).  ``exact`` is the same
computation in plain numpy / torch in 64 bits, with no code of the framework:
labels by Bellman-Ford sweeps over all origins at once, loading by summing the
shortest-path trees, and the Frank-Wolfe iteration of the reference solver
(2^-k step rule, or the exact root with the reverse sweep for the adjoint).
"""

import math

import numpy as np
import torch

from traffic_assignment_gb300 import Solver
from traffic_assignment_gb300.synth import Demand, Network, Scenario

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # one shortest-path tree on a street network: what the `pape` /
        # `sssp_pape` drop-ins do per call (the smallest call, all latency)
        dict(name="tree_street416", mode="sssp", kind="street", rows=16, cols=26, zones=38,
             centroids=False, sources=1, precision="fp64"),
        # labels and predecessors of many origins on a city network
        # (`pape_cuda`, `tapgpu_sssp`)
        dict(name="trees_city10k", mode="sssp", kind="city", rows=100, cols=100, arterials=200,
             zones=1000, demand=1.5e6, centroids=False, sources=100, precision="fp64"),
        # one all-or-nothing loading at given costs (`fw_assign`, `tapgpu_aon`)
        dict(name="load_city10k_fp64", mode="aon", kind="city", rows=100, cols=100, arterials=200,
             zones=1000, demand=1.5e6, centroids=False, precision="fp64"),
        # equilibrium on a 24-node network, every node a zone, fp64 as the
        # drop-in `tap_frankwolfe` runs it
        dict(name="solve_town24_fp64", mode="solve", kind="town", rows=4, cols=6,
             centroids=False, iters=100, warm=False, precision="fp64"),
        # the same on the 416-node street network, fp32 path costs
        dict(name="solve_street416_fp32", mode="solve", kind="street", rows=16, cols=26, zones=38,
             centroids=False, iters=100, warm=False, precision="fp32"),
        # zones as centroids that no path passes through (first thru node)
        dict(name="solve_street454_fp64", mode="solve", kind="street", rows=16, cols=26, zones=38,
             centroids=True, iters=60, warm=False, precision="fp64"),
        # the 10,000-node city with fp32 path costs, restarted from given flows
        # (few iterations: near-ties that fp32 costs break otherwise than fp64
        # ones make the two trajectories part)
        dict(name="solve_city10k_fp32", mode="solve", kind="city", rows=100, cols=100,
             arterials=200, zones=1000, demand=1.5e6, centroids=False, iters=6, warm=True,
             precision="fp32"),
        # the same in fp64 from a cold start
        dict(name="solve_city10k_fp64", mode="solve", kind="city", rows=100, cols=100,
             arterials=200, zones=1000, demand=1.5e6, centroids=False, iters=10, warm=False,
             precision="fp64"),
        # a farm of capacity upgrades in one batch, warm-started (the headline
        # workload, at the batch size one pass affords)
        dict(name="farm_city10k_fp32", mode="farm", kind="city", rows=100, cols=100,
             arterials=200, zones=1000, demand=1.5e6, centroids=False, iters=4, scenarios=64,
             warm=True, precision="fp32"),
        # a farm on a mid-size, not square network in fp64, from a cold start
        dict(name="farm_town3569_fp64", mode="farm", kind="city", rows=43, cols=83, arterials=40,
             zones=101, demand=1.5e5, centroids=False, iters=6, scenarios=37, warm=False,
             precision="fp64"),
        # dVHT/dcapacity through recorded iterations
        dict(name="adjoint_city10k", mode="adjoint", kind="city", rows=100, cols=100,
             arterials=200, zones=1000, demand=1.5e6, centroids=False, iters=10,
             precision="fp64"),
        # a metropolitan network, labels beyond shared memory
        dict(name="solve_metro100k_fp32", mode="solve", kind="city", rows=316, cols=316,
             arterials=2000, zones=1000, demand=4.0e6, centroids=False, iters=3, warm=True,
             precision="fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    precision = rng.choice(["fp32", "fp64"])
    kind = rng.choice(["town", "street", "city", "city", "city"])
    c = dict(kind=kind, centroids=False, precision=precision)
    if kind == "town":
        c.update(rows=rng.randint(2, 7), cols=rng.randint(3, 9))
        nodes = zones = c["rows"] * c["cols"]
    else:
        nodes = _log_int(rng, 100, 4000) if kind == "street" else _log_int(rng, 400, 40000)
        c["rows"] = max(4, int(math.sqrt(nodes) * rng.uniform(0.6, 1.0)))
        c["cols"] = max(5, nodes // c["rows"])
        nodes = c["rows"] * c["cols"]
        lo, hi = (40, 1000) if kind == "city" else (12, 150)
        zones = min(nodes // 4, _log_int(rng, lo, hi))
        c["zones"] = zones
        if kind == "street":
            c["centroids"] = rng.random() < 0.5
        else:
            c["arterials"] = nodes // 50
            c["demand"] = zones * rng.uniform(1500.0, 4000.0)  # congested
    c["mode"] = rng.choice(["sssp", "aon", "solve", "solve", "solve", "farm", "farm", "adjoint"])
    cost = nodes * zones  # path work of one iteration
    if c["mode"] == "sssp":
        c["sources"] = _log_int(rng, 1, max(1, min(300, int(2e6 / nodes))))
    if c["mode"] in ("solve", "adjoint"):
        c["iters"] = max(2, min(rng.randint(3, 60), int(8e7 / cost)))
    if c["mode"] == "farm":
        c["scenarios"] = max(2, min(_log_int(rng, 2, 300), int(1.2e9 / cost / 2)))
        c["iters"] = max(2, min(rng.randint(2, 12), int(1.2e9 / cost / c["scenarios"])))
    if c["mode"] in ("solve", "farm"):
        c["warm"] = rng.random() < 0.5
    if kind == "city" and precision == "fp32":  # (see solve_city10k_fp32)
        if c["mode"] == "adjoint":
            c["precision"] = "fp64"
        elif "iters" in c:
            c["iters"] = min(c["iters"], 6 if c["warm"] else 2)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _grid_streets(rows, cols):
    i = np.arange(rows * cols).reshape(rows, cols)
    return np.concatenate([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                           np.stack([i[:-1].ravel(), i[1:].ravel()], 1)])


def _tree_mask(rng, n, streets):
    """A random spanning tree of the streets (Kruskal in random order)."""
    root = list(range(n))

    def find(a):
        while root[a] != a:
            root[a] = root[root[a]]
            a = root[a]
        return a

    keep = np.zeros(len(streets), bool)
    for i in rng.permutation(len(streets)):
        a, b = find(int(streets[i, 0])), find(int(streets[i, 1]))
        if a != b:
            root[a] = b
            keep[i] = True
    return keep


def _inputs(case, seed):
    """(Network, Demand) of the case, from the seed."""
    rng = np.random.default_rng([seed, 77])
    rows, cols = case["rows"], case["cols"]
    n = rows * cols
    streets = _grid_streets(rows, cols)
    px = np.arange(n) % cols + rng.uniform(-0.3, 0.3, n)
    py = np.arange(n) // cols + rng.uniform(-0.3, 0.3, n)
    if case["kind"] == "street":
        keep = _tree_mask(rng, n, streets)
        spare = np.nonzero(~keep)[0]
        keep[rng.choice(spare, min(len(spare), max(1, n // 10)), replace=False)] = True
        streets = streets[keep]
    u = np.concatenate([streets[:, 0], streets[:, 1]])
    v = np.concatenate([streets[:, 1], streets[:, 0]])
    m = len(u)
    mean_log = math.log(1.5) - 0.18
    if case["kind"] == "town":
        fft, cap = rng.uniform(2.0, 10.0, m), rng.uniform(4000.0, 26000.0, m)
    elif case["kind"] == "street":
        fft, cap = rng.lognormal(mean_log, 0.6, m), rng.uniform(1000.0, 8000.0, m)
    else:
        fft = rng.lognormal(mean_log, 0.6, m)
        cap = rng.choice([1800.0, 3600.0], m, p=[0.7, 0.3])
        # long two-way arterials over 6 to 30 blocks, faster per block
        k = case["arterials"]
        a = rng.integers(0, n, 2 * k)
        dr, dc = rng.integers(-15, 16, 2 * k), rng.integers(-15, 16, 2 * k)
        b = (np.clip(a // cols + dr, 0, rows - 1) * cols + np.clip(a % cols + dc, 0, cols - 1))
        blocks = np.abs(a // cols - b // cols) + np.abs(a % cols - b % cols)
        lo, hi = np.minimum(a, b)[blocks >= 6], np.maximum(a, b)[blocks >= 6]
        _, first = np.unique(lo * n + hi, return_index=True)
        first = np.sort(first)[:k]
        lo, hi, blocks = lo[first], hi[first], blocks[blocks >= 6][first]
        afft = 0.45 * 1.5 * blocks * rng.lognormal(0.0, 0.15, len(lo))
        u, v = np.concatenate([u, lo, hi]), np.concatenate([v, hi, lo])
        fft = np.concatenate([fft, afft, afft * rng.uniform(0.97, 1.03, len(lo))])
        cap = np.concatenate([cap, np.full(2 * len(lo), 7200.0)])
    z = n if case["kind"] == "town" else case["zones"]
    zone_at = rng.permutation(n) if z == n else rng.choice(n, z, replace=False)
    number = np.zeros(n, np.int64)
    if case["centroids"]:  # zones 1..z tied to street nodes z+1..z+n by connectors
        number[:] = np.arange(z + 1, z + n + 1)
        init, term = number[u], number[v]
        zid, at = np.arange(1, z + 1), number[zone_at]
        init, term = np.concatenate([init, zid, at]), np.concatenate([term, at, zid])
        fft = np.concatenate([fft, np.full(2 * z, 0.05)])
        cap = np.concatenate([cap, np.full(2 * z, 50000.0)])
        nodes, first_thru = n + z, z + 1
    else:
        rest = np.ones(n, bool)
        rest[zone_at] = False
        number[zone_at] = np.arange(1, z + 1)
        number[rest] = np.arange(z + 1, n + 1)
        init, term, nodes, first_thru = number[u], number[v], n, 1
    order = np.lexsort((term, init))
    m = len(order)
    net = Network(num_nodes=nodes, num_zones=z, first_thru_node=first_thru,
                  init=init[order], term=term[order], capacity=cap[order], length=np.ones(m),
                  fft=fft[order], alpha=np.full(m, 0.15), beta=np.full(m, 4.0),
                  speed=np.zeros(m), toll=np.zeros(m), link_type=np.ones(m, np.int16))
    if case["kind"] == "city":
        x, y = px[zone_at], py[zone_at]
        t = (rng.lognormal(0.0, 0.5, z)[:, None] * rng.lognormal(0.0, 0.5, z)[None, :] *
             np.exp(-np.hypot(x[:, None] - x[None], y[:, None] - y[None]) /
                    (0.2 * max(rows, cols))))
        np.fill_diagonal(t, 0.0)
        t *= case["demand"] / t.sum()
    elif case["kind"] == "street":
        t = np.where(rng.random((z, z)) < 0.30, rng.uniform(1.0, 500.0, (z, z)), 0.0)
        np.fill_diagonal(t, 0.0)
    else:
        t = rng.integers(0, 2001, (z, z)).astype(np.float64)
        np.fill_diagonal(t, 0.0)
    o, d = np.nonzero(t) if case["kind"] != "town" else np.divmod(np.arange(z * z), z)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(o + 1, minlength=z + 1))])
    dem = Demand(num_zones=z, od_ptr=ptr.astype(np.int64), od_dest=(d + 1).astype(np.int64),
                 od_demand=t[o, d])
    return net, dem


def _warm_flows(net, seed):
    """Flows of a loaded network to restart from: most links below capacity,
    some above it."""
    rng = np.random.default_rng([seed, 78])
    return net.capacity * np.minimum(rng.lognormal(-0.7, 0.6, net.num_links), 1.8)


def _link_costs(net, seed):
    x = _warm_flows(net, seed + 1)
    return net.fft * (1.0 + net.alpha * (x / net.capacity) ** net.beta)


def _sources(case, net, seed):
    rng = np.random.default_rng([seed, 79])
    k = case["sources"]
    return rng.choice(np.arange(1, net.num_nodes + 1), k, replace=k > net.num_nodes)


def _upgrades(case, net, seed):
    """Scenario s raises the capacity of 1 to 20 links by 25 to 100 %."""
    rng = np.random.default_rng([seed, 80])
    out = []
    for s in range(case["scenarios"]):
        k = int(rng.integers(1, min(20, net.num_links) + 1))
        links = np.sort(rng.choice(net.num_links, k, replace=False)).astype(np.int64)
        out.append(Scenario(f"s{s:04d}", links,
                            net.capacity[links] * (1.0 + rng.uniform(0.25, 1.0, k))))
    return out


def prepare(case, seed):
    """The handle and the arrays a program holds before the call."""
    net, dem = _inputs(case, seed)
    mode = case["mode"]
    st = dict(mode=mode, iters=case.get("iters", 0))
    if mode == "adjoint":
        st["solver"] = Solver(net, dem, precision=case["precision"], record_tape=True,
                              tape_capacity=case["iters"], line_search="exact")
        rng = np.random.default_rng([seed, 81])
        st["capacity"] = net.capacity * rng.uniform(0.9, 1.3, net.num_links)
        return st
    st["solver"] = Solver(net, dem, precision=case["precision"])
    if mode in ("sssp", "aon"):
        st["costs"] = _link_costs(net, seed)
    if mode == "sssp":
        st["sources"] = _sources(case, net, seed)
    if mode in ("solve", "farm"):
        st["x0"] = _warm_flows(net, seed) if case["warm"] else None
    if mode == "farm":
        st["upgrades"] = _upgrades(case, net, seed)
    return st


_SCALARS = ("objective", "relgap", "total_cost", "avg_excess", "lambda_last")


def run(state):
    """One call as a program makes it, and all it returns."""
    s, mode = state["solver"], state["mode"]
    if mode == "sssp":
        dist, pred = s.sssp(state["costs"], state["sources"])
        return dict(dist=dist, pred=pred)
    if mode == "aon":
        return s.aon(state["costs"])
    if mode == "solve":
        r = s.solve(max_iters=state["iters"], x0=state["x0"])
        volume, cost = s.flows()
        return dict(volume=volume, cost=cost, iterations=r["iterations"],
                    **{k: r[k] for k in _SCALARS})
    if mode == "farm":
        rs = s.solve_scenarios(state["upgrades"], max_iters=state["iters"], x0=state["x0"])
        volume, cost = s.flows_batch()
        return dict(volume=volume, cost=cost,
                    iterations=np.array([r["iterations"] for r in rs]),
                    **{k: np.array([r[k] for r in rs]) for k in _SCALARS})
    s.set_capacity(state["capacity"])  # adjoint
    s.solve(max_iters=state["iters"])
    vht, grad = s.adjoint_vht()
    return dict(vht=vht, grad=grad)


def work(case):
    """What one pass cannot do without: the network, demand, warm start and
    edits read once, the results written once; two operations (an addition and
    a comparison) per link and origin of every shortest-path solution, one
    addition per node and origin of every loading, and the link formulas."""
    n = case["rows"] * case["cols"]
    z = n if case["kind"] == "town" else case["zones"]
    if case["kind"] == "street":
        m = 2 * (n - 1 + n // 10)
    else:
        m = 2 * (case["rows"] * (case["cols"] - 1) + case["cols"] * (case["rows"] - 1))
        m += 2 * case.get("arterials", 0)
    if case["centroids"]:
        n, m = n + z, m + 2 * z
    nnz = z * z * (0.3 if case["kind"] == "street" else 1.0)
    topo, params, demand = 8.0 * m, 32.0 * m, 12.0 * nnz
    mode = case["mode"]
    if mode == "sssp":
        k = case["sources"]
        return dict(bytes=topo + 8.0 * m + 16.0 * k * (n + 1), flops=2.0 * k * m)
    per_iter = z * (2.0 * m + n)
    if mode == "aon":
        return dict(bytes=topo + 16.0 * m + demand, flops=per_iter)
    iters = case["iters"]
    per_iter += 80.0 * m  # objective, 12 or more line-search candidates, cost update
    if mode == "farm":
        k = case["scenarios"]
        return dict(bytes=topo + params + demand + 8.0 * m + k * (160.0 + 16.0 * m),
                    flops=k * iters * per_iter)
    extra = 60.0 * m * iters if mode == "adjoint" else 0.0
    return dict(bytes=topo + params + demand + 24.0 * m,
                flops=(iters + 1) * per_iter + extra)


# ---------------------------------------------------------------------------
# the same in 64 bits, without the framework
# ---------------------------------------------------------------------------


class _Paths:
    """Shortest paths and loading of all origins of one network at once."""

    def __init__(self, net, dem):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n1, self.m, self.thru = net.num_nodes + 1, net.num_links, net.first_thru_node
        tail, head = torch.as_tensor(net.init), torch.as_tensor(net.term)
        order = torch.sort(head, stable=True).indices
        deg = torch.bincount(head, minlength=self.n1)
        start = torch.cumsum(deg, 0) - deg
        rank = torch.arange(self.m) - start[head[order]]
        self.layers = []  # the j-th in-link of every node that has more than j
        for j in range(int(deg.max())):
            k = order[rank == j]
            self.layers.append([t.to(self.dev) for t in (k, tail[k], head[k])])
        self.tail = tail.to(self.dev)
        if dem is not None:
            z = dem.num_zones
            o = np.repeat(np.arange(z), np.diff(dem.od_ptr[1:z + 2]))
            q = np.where(dem.od_dest == o + 1, 0.0, np.maximum(dem.od_demand, 0.0))
            demand = torch.zeros((self.n1, z), dtype=torch.float64)
            demand.index_put_((torch.as_tensor(dem.od_dest), torch.as_tensor(o)),
                              torch.as_tensor(q), accumulate=True)
            self.demand, self.origins = demand.to(self.dev), torch.arange(1, z + 1)

    def labels(self, w, sources):
        """[n1][sources]: sweeps over every in-link until nothing improves."""
        w = torch.as_tensor(w, dtype=torch.float64).to(self.dev)
        src = torch.as_tensor(sources).to(self.dev)
        cols = torch.arange(len(src), device=self.dev)
        d = torch.full((self.n1, len(src)), math.inf, dtype=torch.float64, device=self.dev)
        d[src, cols] = 0.0
        for sweep in range(self.n1 + 1):
            last = d.clone() if sweep % 8 == 0 else None
            for k, t, h in self.layers:
                cand = d[t] + w[k][:, None]
                self._closed(cand, t, src)
                d[h] = torch.minimum(d[h], cand)
            if last is not None and torch.equal(last, d):
                return d
        return d

    def _closed(self, cand, t, src):
        """Nodes below the first thru node are only left by their own origin."""
        if self.thru > 1:
            cand.masked_fill_((t[:, None] < self.thru) & (src[None] != t[:, None]), math.inf)

    def load(self, w):
        """All-or-nothing link volumes at costs w."""
        wd = torch.as_tensor(w, dtype=torch.float64).to(self.dev)
        src = self.origins.to(self.dev)
        d = self.labels(w, self.origins)
        best = torch.full_like(d, math.inf)
        link = torch.full(d.shape, -1, dtype=torch.int32, device=self.dev)
        for k, t, h in self.layers:
            cand = d[t] + wd[k][:, None]
            self._closed(cand, t, src)
            cand[d[t] >= d[h]] = math.inf
            better = cand < best[h]
            best[h] = torch.where(better, cand, best[h])
            link[h] = torch.where(better, k[:, None].to(torch.int32), link[h])
        del best, d
        z = len(src)
        cols = torch.arange(z, device=self.dev)
        link[src, cols] = -1
        # subtree totals by doubling: after step i a node has the demand of its
        # descendants fewer than 2^i links below
        flat = torch.arange(self.n1 * z, device=self.dev).view(self.n1, z)
        up = torch.where(link >= 0, self.tail[link.clamp(min=0).long()] * z + cols, flat)
        total, moving = self.demand.clone().flatten(), link >= 0
        up, moving = up.flatten(), moving.flatten()
        while bool(moving.any()):
            add = torch.zeros_like(total)
            add.index_add_(0, up[moving], total[moving])
            total = total + add
            moving = moving & moving[up]
            up = up[up]
        has = link.flatten() >= 0
        y = torch.zeros(self.m, dtype=torch.float64, device=self.dev)
        y.index_add_(0, link.flatten()[has].long(), total[has])
        return y.cpu().numpy()


def _cost(net, cap, x):
    return net.fft * (1.0 + net.alpha * (x / cap) ** net.beta)


def _dcost(net, cap, x):
    return net.fft * net.alpha * net.beta * (x / cap) ** (net.beta - 1.0) / cap


def _equilibrate(net, paths, total, cap, x, iters, exact_step, tape=None):
    """Frank-Wolfe iterations from the flows x (None: loaded at free flow)."""
    x = paths.load(net.fft) if x is None else x.copy()
    t = _cost(net, cap, x)
    best, r = -math.inf, {}
    for _ in range(iters):
        y = paths.load(t)
        d = y - x

        def slope(lam):
            return float(np.dot(_cost(net, cap, x + lam * d), d))

        g0 = float(np.dot(t, d))
        obj = float(np.sum(x * net.fft * (1.0 + net.alpha / (net.beta + 1.0) *
                                          (x / cap) ** net.beta)))
        best = max(best, obj + g0)
        lam = 0.0
        if g0 < 0:
            lam = 1.0
            if slope(1.0) > 0:
                if exact_step:
                    lo, hi = 0.0, 1.0
                    for _ in range(200):
                        mid = 0.5 * (lo + hi)
                        if mid <= lo or mid >= hi:
                            break
                        lo, hi = (lo, mid) if slope(mid) > 0 else (mid, hi)
                    lam = 0.5 * (lo + hi)
                else:
                    lam = 0.5
                    while slope(lam) > 0:
                        lam *= 0.5
        if tape is not None:
            tape.append((x, d, lam))
        r = dict(objective=obj, relgap=(obj - best) / abs(best), avg_excess=-g0 / total,
                 lambda_last=lam)
        x = x + lam * d
        t = _cost(net, cap, x)
    r["total_cost"] = float(np.dot(x, t))
    return x, t, r


def exact(case, seed):
    net, dem = _inputs(case, seed)
    mode = case["mode"]
    if mode == "sssp":
        p = _Paths(net, None)
        d = p.labels(_link_costs(net, seed), _sources(case, net, seed)).T.cpu().numpy()
        return dict(dist=np.where(np.isinf(d), np.finfo(np.float64).max, d), pred=None)
    paths = _Paths(net, dem)
    if mode == "aon":
        return paths.load(_link_costs(net, seed))
    total, iters = float(dem.od_demand.sum()), case["iters"]
    if mode == "solve":
        x, t, r = _equilibrate(net, paths, total, net.capacity,
                               _warm_flows(net, seed) if case["warm"] else None, iters, False)
        return dict(volume=x, cost=t, iterations=iters, **{k: r[k] for k in _SCALARS})
    if mode == "farm":
        x0 = _warm_flows(net, seed) if case["warm"] else paths.load(net.fft)
        xs, ts, rs = [], [], []
        for sc in _upgrades(case, net, seed):
            cap = net.capacity.copy()
            cap[sc.links] = sc.new_capacity
            x, t, r = _equilibrate(net, paths, total, cap, x0, iters, False)
            xs.append(x)
            ts.append(t)
            rs.append(r)
        return dict(volume=np.stack(xs), cost=np.stack(ts),
                    iterations=np.full(len(rs), iters),
                    **{k: np.array([r[k] for r in rs]) for k in _SCALARS})
    rng = np.random.default_rng([seed, 81])
    cap = net.capacity * rng.uniform(0.9, 1.3, net.num_links)
    tape = []
    x, t, r = _equilibrate(net, paths, total, cap, None, iters, True, tape)
    beta = net.beta
    xbar = t + x * _dcost(net, cap, x)
    cbar = -x * net.fft * net.alpha * beta * (x / cap) ** beta / cap
    for xk, d, lam in reversed(tape):  # the loads held fixed, the step by the implicit rule
        q = xk + lam * d
        if 0.0 < lam < 1.0:
            coef = -float(np.dot(xbar, d)) / float(np.dot(_dcost(net, cap, q), d * d))
            cbar = cbar + coef * (-net.fft * net.alpha * beta * (q / cap) ** beta / cap) * d
            xbar = (1.0 - lam) * xbar + coef * (_dcost(net, cap, q) * (1.0 - lam) * d -
                                                _cost(net, cap, q))
        else:
            xbar = (1.0 - lam) * xbar
    return dict(vht=r["total_cost"], grad=cbar)
