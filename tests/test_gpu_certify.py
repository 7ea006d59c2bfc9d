"""Proof that a component is its own densest set, against the flow search: the
same answers whether a context may use the proof (the default) or has to run its
flows (64-bit flow state asked for), on components around one word of vertices,
many words, the largest the proof takes and past it, on several components of one
graph, on batches, and where a subset is denser than the whole by little."""
import math

import numpy as np
import pytest

import cds_b200 as cds
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def both():
    with cds.Context(0) as a, cds.Context(0, flags=cds.CONFIG_WIDE_FLOW) as b:
        yield a, b


def answer(c, off, adj, k, **kw):
    g = c.graph(off, adj)
    s = c.solve(g, k, **kw)
    g.free()
    return (s.num, s.den, s.vertices.tolist(), s.upper_bound, s.n_components, s.pruned_edges, s.core_cliques,
            s.early_stopped)


def dense(n, p, seed):
    off, adj = cds.gen_er(n, 0.0, 1)
    off, adj, _ = cds.gen_plant(off, adj, n, p, seed)
    return off, adj


@pytest.mark.parametrize("k", [2, 3, 4, 5])
@pytest.mark.parametrize("n,p", [(6, 1.0), (31, 0.6), (32, 0.6), (33, 0.6), (65, 0.5), (127, 0.4), (129, 0.35)])
def test_one_dense_component(both, n, p, k):
    off, adj = dense(n, p, n + k)
    a, b = (answer(c, off, adj, k) for c in both)
    assert a == b
    o = oracle.solve(off, adj, k)
    assert a[0] * o["den"] == o["num"] * a[1]


@pytest.mark.parametrize("k,n,p", [(2, 1023, 0.05), (2, 1024, 0.05), (2, 1025, 0.05), (3, 1024, 0.06), (3, 1025, 0.06),
                                   (4, 700, 0.12)])
def test_large_components(both, k, n, p):
    off, adj = dense(n, p, 5)
    a, b = (answer(c, off, adj, k) for c in both)
    assert a == b


@pytest.mark.parametrize("k", [2, 3, 4, 5])
@pytest.mark.parametrize("seed", range(4))
def test_sparse_and_skewed(both, seed, k):
    off, adj = cds.gen_rmat(10, 6.0, seed)
    if seed % 2:
        off, adj, _ = cds.gen_plant(off, adj, 30, 0.5, seed)
    for search in ("dinkelbach", "bisect"):
        a, b = (answer(c, off, adj, k, search=search) for c in both)
        assert a == b


@pytest.mark.parametrize("k", [2, 3, 4])
def test_several_components_and_ties(both, k):
    # copies of one dense block beside denser and sparser ones
    parts = [dense(40, 0.5, 1), dense(40, 0.5, 1), dense(40, 0.5, 2), dense(24, 0.8, 3), dense(24, 0.8, 3)]
    u, v, base = [], [], 0
    for off, adj in parts:
        n = len(off) - 1
        u.append(np.repeat(np.arange(n), np.diff(off.astype(np.int64))) + base)
        v.append(adj.astype(np.int64) + base)
        base += n
    off, adj = cds.csr_from_edges(base, np.concatenate(u), np.concatenate(v))
    a, b = (answer(c, off, adj, k) for c in both)
    assert a == b


@pytest.mark.parametrize("k", [2, 3])
def test_a_subset_barely_denser(both, k):
    # a circulant graph is its own densest set; one chord more makes a proper
    # subset of nothing, one vertex less attached makes a subset denser
    n = 60
    ring = np.arange(n)
    for drop in (0, 1, 2):
        u, v = [], []
        for d in range(1, 5):
            u.append(ring)
            v.append((ring + d) % n)
        u, v = np.concatenate(u), np.concatenate(v)
        keep = ~((u == 0) & (v <= drop))
        off, adj = cds.csr_from_edges(n, u[keep], v[keep])
        a, b = (answer(c, off, adj, k) for c in both)
        assert a == b
        o = oracle.solve(off, adj, k)
        assert (a[0], a[1]) == (o["num"], o["den"]) and a[2] == o["vertices"].tolist()


def test_batches(both):
    rng = np.random.default_rng(3)
    graphs = []
    for i in range(40):
        n = int(rng.integers(30, 900))
        off, adj = cds.gen_er(n, float(rng.uniform(4, 12)) / n, i)
        off, adj, _ = cds.gen_plant(off, adj, int(rng.integers(10, 30)), 0.6, i)
        graphs.append((off, adj, int(rng.integers(2, 6))))
    got = []
    for c in both:
        gs = [(c.graph(off, adj), k) for off, adj, k in graphs]
        got.append([(s.num, s.den, s.vertices.tolist(), s.upper_bound)
                    for s in c.solve_batch([(g, cds.make_params(k)) for g, k in gs])])
        for g, _ in gs:
            g.free()
    assert got[0] == got[1]


def test_units_of_many_cliques(both):
    # an edge of the complete graph on 560 vertices has 155,403 4-cliques before its
    # later neighbours': k 2^46 units of each pass 64 bits
    n, k = 560, 4
    off, adj = dense(n, 1.0, 1)
    g = both[0].graph(off, adj)
    s = both[0].solve(g, k)
    g.free()
    assert s.num * n == math.comb(n, k) * s.den
    assert s.vertices.tolist() == list(range(n))


@pytest.mark.parametrize("k", [2, 3, 4])
def test_cores_of_a_batch_side_by_side(both, k):
    # every core within its own rows, however many vertices they have together (with
    # k = 2 one core is wider than any other and past the proof's size)
    rng = np.random.default_rng(7)
    graphs = [cds.gen_rmat(12, float(rng.uniform(6, 12)), i) for i in range(24)]
    graphs.insert(5, cds.gen_er(5000, 12.0 / 5000, 3))
    graphs.insert(0, cds.gen_er(40, 0.0, 4))  # no clique at all
    gs = [both[0].graph(*g) for g in graphs]
    params = cds.make_params(k)
    got = both[0].solve_batch([(g, params) for g in gs])
    for g, b in zip(gs, got):
        s = both[0].solve(g, k)
        assert (s.num, s.den, s.vertices.tolist(), s.pruned_edges, s.n_components, s.core_size) == (
            b.num, b.den, b.vertices.tolist(), b.pruned_edges, b.n_components, b.core_size)
        g.free()
    assert k == 4 or sum(b.core_size for b in got) > 4096


def two_rings(n, near, nearer, seed):
    """Two rings of n / 2 vertices on mixed ids, one whose vertices are adjacent up to
    distance `near`, one up to `nearer` < `near` - 1; ten vertices of the second are
    joined to two neighbours of the first.  The first is the only densest set."""
    size, rng = n // 2, np.random.default_rng(seed)
    u, v = [], []
    for first, m, reach in ((0, size, near), (size, n - size, nearer)):
        for d in range(1, reach + 1):
            u.append(first + np.arange(m))
            v.append(first + (np.arange(m) + d) % m)
    spread = np.arange(10) * (size // 10)
    u += [spread, spread + 1]
    v += [size + spread, size + spread]
    ids = rng.permutation(n)
    off, adj = cds.csr_from_edges(n, ids[np.concatenate(u)], ids[np.concatenate(v)])
    return off, adj, np.sort(ids[:size])


# components of a whole block of 1,024 threads, and some of whose last warp is partly or
# wholly idle: the scan over the order's ranks spans up to 32 warps
@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("n", [700, 992, 993, 1000, 1023, 1024])
def test_a_denser_subset_of_a_large_component(both, n, k):
    off, adj, ring = two_rings(n, 12, 9, n + k)
    proof = both[0]
    proof.profile(True)
    proof.profile_read()
    a = answer(proof, off, adj, k)
    launches = proof.profile_read()
    proof.profile(False)
    assert a == answer(both[1], off, adj, k)
    assert a[0] == len(ring) * {2: 12, 3: 66}[k] and a[2] == ring.tolist()
    assert a[4] == 1  # in one component with the other ring, and no flow was needed
    assert "certify" in launches and "push_relabel" not in launches


def test_warm_start_by_the_networks_left(ctx):
    # a network that the proof never saw (more than 1,024 vertices, few cliques) starts
    # without a split, whatever else of its batch was proved
    large = cds.gen_er(3000, 60.0 / 2999, 12)
    small = cds.gen_plant(*cds.gen_er(2000, 0.004, 0), 40, 0.6, 0)[:2]
    launches = []
    for graphs in ((large,), (large, small)):
        gs = [ctx.graph(off, adj) for off, adj in graphs]
        ctx.profile(True)
        ctx.profile_read()
        ctx.solve_batch([(g, cds.make_params(3)) for g in gs])
        launches.append(ctx.profile_read())
        ctx.profile(False)
        for g in gs:
            g.free()
    assert all("push_relabel" in x and "flow_warm" not in x for x in launches)
    assert "certify" in launches[1] and "certify" not in launches[0]
