"""The work a user of cds_b200 has it do, as cases to be timed.

Each case is one pass through the package's public entry points on seeded
synthetic graphs: whole solves from the smallest graph to the largest, the
listing and clique-core stages by themselves, a batch of unequal instances
and a burst of served requests that bring their graphs with them.

listed()  the cases
draw()    one more case of the same ranges
prepare() the inputs of a case, made from the seed
run()     one pass
work()    the bytes a pass cannot do without
exact()   the answers of small counting cases by plain numpy
"""
import math

import numpy as np
import torch

import cds_b200 as cds

# One context serves the process, as in a user's program; the request server
# has its own, with the device memory it may fill.
_SERVE_BUDGET = 40 << 30
_shared = {}


def _context():
    if "ctx" not in _shared:
        _shared["ctx"] = cds.Context(0)
    return _shared["ctx"]


def _server():
    if "server" not in _shared:
        _shared["server_ctx"] = cds.Context(0, mem_budget=_SERVE_BUDGET)
        _shared["server"] = _shared["server_ctx"].server(max_batch=64, mem_budget=_SERVE_BUDGET, max_inflight=4)
    return _shared["server"]


def _case(name, kind, graph, n, degree, plant, k, search="dinkelbach"):
    """degree: average degree asked of the generator (R-MAT drops duplicates
    and self-loops); plant: size of a planted community of edge probability
    one half (0: none)."""
    c = {"kind": kind, "graph": graph, "n": n, "degree": degree, "plant": plant, "k": k, "search": search}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest solve: a sparse random graph with a small community in
        # it, where kernel launches and host waits count for most
        _case("solve-er-2k-k3", "solve", "er", 2000, 8.0, 40, 3),
        # R-MAT scale 14, edge factor 8 at each clique size of the benchmark:
        # edges, triangles, 4-cliques
        _case("solve-rmat-16k-k2", "solve", "rmat", 16384, 16.0, 0, 2),
        _case("solve-rmat-16k-k3", "solve", "rmat", 16384, 16.0, 0, 3),
        _case("solve-rmat-16k-k4", "solve", "rmat", 16384, 16.0, 0, 4),
        # a large sparse graph with few cliques: the largest Erdos-Renyi
        # instance of the batched configuration, solved alone
        _case("solve-er-50k-k3", "solve", "er", 49999, 24.0, 130, 3),
        # a large skewed graph of odd size at the common clique size: the
        # largest request of the served configuration
        _case("solve-rmat-200k-k3", "solve", "rmat", 199999, 24.0, 0, 3),
        # the largest solve: R-MAT scale 18, edge factor 16, planted community
        # of 300, 4-cliques in the billions
        _case("solve-rmat-262k-k4", "solve", "rmat", 262144, 32.0, 300, 4),
        # clique sizes past the specialised ones (enumeration by depth-first
        # search), on a graph of odd size
        _case("solve-rmat-8k-k5", "solve", "rmat", 8191, 12.0, 0, 5),
        # the clique-core numbers of every vertex, for a caller who wants the
        # decomposition and no densest subgraph
        _case("core-rmat-65k-k4", "core", "rmat", 65536, 24.0, 0, 4),
        # counting alone: the clique total and every vertex's clique degree
        _case("list-rmat-262k-k4", "list", "rmat", 262144, 32.0, 0, 4),
        # instances of unequal size and clique size in one call, sized as the
        # batched configuration draws them
        {"name": "batch-48", "kind": "batch", "count": 48, "lo": 500, "hi": 50000, "mix": 2},
        # requests that arrive together, each with its graph in host memory
        # (upload and checks included), answered by a running server
        {"name": "serve-24", "kind": "serve", "count": 24, "lo": 1000, "hi": 50000, "mix": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "core", "list", "batch", "serve"])
    if kind in ("batch", "serve"):
        return {"kind": kind, "count": rng.randint(8, 48 if kind == "batch" else 24),
                "lo": 500 if kind == "batch" else 1000, "hi": rng.randint(10000, 50000), "mix": rng.randint(0, 1 << 20)}
    graph = rng.choice(["er", "rmat"])
    k = rng.choice([2, 3, 3, 4, 4, 5])
    # deep cliques multiply with the size of a skewed graph: keep those small
    n = _log_uniform(rng, 1000, 8191 if k == 5 else 200000)
    degree = round(rng.uniform(6.0, 12.0 if k == 5 else 24.0), 2)
    plant = rng.randint(20, 60 if k == 5 else 200)
    if graph == "rmat" and rng.random() < 0.5:  # dense by itself; a random graph has few cliques but the planted ones
        plant = 0
    search = rng.choice(["dinkelbach", "dinkelbach", "core", "bisect"]) if kind == "solve" else "dinkelbach"
    return _case(None, kind, graph, n, degree, plant, k, search)


def _graph(graph, n, degree, plant, seed):
    if graph == "er":
        off, adj = cds.gen_er(n, degree / (n - 1), seed)
    else:
        scale = max(1, (n - 1).bit_length())
        off, adj = cds.gen_rmat(scale, degree / 2 * n / (1 << scale), seed, n=n)
    if plant:
        off, adj, _ = cds.gen_plant(off, adj, min(plant, n), 0.5, seed + 17)
    return off, adj


def _host_graph(case, seed):
    return _graph(case["graph"], case["n"], case["degree"], case["plant"], seed * 1000003 + 1)


def _mix(case):
    """(graph, n, degree, plant, k) of each instance of a batch or a burst; the
    sizes belong to the case, the graphs to the seed."""
    rng = np.random.default_rng(case["mix"])
    shapes = []
    for i in range(case["count"]):
        n = int(round(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"])))))
        if case["kind"] == "batch":
            shapes.append(("er" if i % 2 == 0 else "rmat", n, float(rng.uniform(4, 32)), int(rng.integers(20, 201)),
                           int(rng.integers(2, 5))))
        else:
            shapes.append(("rmat", n, float(rng.uniform(8, 32)), 0, 3 if rng.random() < 0.75 else 4))
    return shapes


def prepare(case, seed):
    seed = int(seed)
    if case["kind"] == "batch":
        ctx = _context()
        return {"kind": "batch", "ctx": ctx, "jobs": [
            (ctx.graph(*_graph(*shape, seed * 100003 + i)), cds.make_params(k)) for i, (*shape, k) in enumerate(_mix(case))]}
    if case["kind"] == "serve":
        requests = []
        for i, (*shape, k) in enumerate(_mix(case)):
            off, adj = _graph(*shape, seed * 7919 + i)
            requests.append((torch.from_numpy(off.view(np.int64)).pin_memory(),
                             torch.from_numpy(adj.view(np.int32)).pin_memory(), shape[1], cds.make_params(k)))
        return {"kind": "serve", "server": _server(), "requests": requests}
    ctx = _context()
    off, adj = _host_graph(case, seed)
    return {"kind": case["kind"], "ctx": ctx, "g": ctx.graph(off, adj), "k": case["k"], "search": case["search"]}


def _answer(s, n):
    """A solution as numbers and arrays: the answer (its vertices as a mask over
    the graph's n), its bound, and what every stage on the way reports."""
    inside = np.zeros(n, np.uint8)
    inside[s.vertices] = 1
    return {
        "density": np.array([s.num, s.den], np.int64),
        "vertices": inside,
        "upper_bound": np.array(s.upper_bound, np.int64),
        "cliques": s.total_cliques,
        "core": np.array([s.max_core, s.core_threshold, *s.core_density, s.core_size, s.core_cliques], np.int64),
        "shape": np.array([s.pruned_edges, s.n_components, s.peel_levels], np.int64),
    }


def _joined(solutions, sizes):
    """Many solutions as one set of arrays, in order (a list of them each would
    be hundreds of outputs)."""
    each = [_answer(s, n) for s, n in zip(solutions, sizes)]
    return {key: np.concatenate([np.atleast_1d(a[key]) for a in each]) for key in each[0]}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return _answer(state["ctx"].solve(state["g"], state["k"], search=state["search"]), state["g"].n)
    if kind == "core":
        core, largest, count = state["ctx"].clique_core(state["g"], state["k"])
        return {"core": core, "max_core": largest, "cliques": count}
    if kind == "list":
        count, degree = state["ctx"].list_cliques(state["g"], state["k"])
        return {"cliques": count, "degree": degree}
    if kind == "batch":
        return _joined(state["ctx"].solve_batch(state["jobs"]), [g.n for g, _ in state["jobs"]])
    server = state["server"]
    tickets = [server.submit_csr(off.data_ptr(), adj.data_ptr(), n, p) for off, adj, n, p in state["requests"]]
    return _joined([server.wait(t) for t in tickets], [n for _, _, n, _ in state["requests"]])


def work(case):
    """The graph read once and the answer written once: 8 bytes an offset and
    4 an arc; a count or core number per vertex where the pass returns them.
    What the cliques themselves cost depends on how they are counted, so they
    are not in it."""
    if case["kind"] in ("batch", "serve"):
        return {"bytes": sum(8 * (n + 1) + 4 * (n * degree + 0.5 * plant * plant) + 200 + n
                             for _, n, degree, plant, _ in _mix(case)), "flops": 0}
    n = case["n"]
    arcs = n * case["degree"] + 0.5 * case["plant"] * max(0, case["plant"] - 1)
    out = 8 * n if case["kind"] in ("core", "list") else 200 + n
    return {"bytes": 8 * (n + 1) + 4 * arcs + out, "flops": 0}


def _cliques_of(adjacent, size):
    """Cliques of `size` vertices of a graph given as a dense 0/1 matrix: their
    number, and how many hold each vertex."""
    n = len(adjacent)
    if size == 1:
        return n, np.ones(n, np.int64)
    if size == 2:
        degree = adjacent.sum(1)
        return int(degree.sum()) // 2, degree
    if size == 3:
        degree = ((adjacent @ adjacent) * adjacent).sum(1) / 2
        return int(degree.sum()) // 3, degree
    degree = np.zeros(n, np.int64)
    for v in range(n):
        near = np.flatnonzero(adjacent[v])
        if len(near) >= size - 1:
            degree[v] = _cliques_of(adjacent[np.ix_(near, near)], size - 1)[0]
    return int(degree.sum()) // size, degree


def exact(case, seed):
    """The counting cases of up to 4,000 vertices by dense matrices in 64 bits
    (every value below 2^53); the others have no short plain form."""
    if case["kind"] != "list" or case["n"] > 4000:
        return None
    off, adj = _host_graph(case, int(seed))
    n = case["n"]
    adjacent = np.zeros((n, n))
    adjacent[np.repeat(np.arange(n), np.diff(off.astype(np.int64))), adj] = 1
    count, degree = _cliques_of(adjacent, case["k"])
    return {"cliques": count, "degree": degree.astype(np.uint64)}
