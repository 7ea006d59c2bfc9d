"""Clique-core numbers by weighted arcs: exact against the oracle's peel where rows
are handled by warps and by blocks, and against known values where a vertex has
more later neighbours than one team counts (a hub of low core number among
vertices of higher ones)."""
from math import comb

import numpy as np
import pytest

import cds_b200 as cds
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with cds.Context(0) as c:
        yield c


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6])
@pytest.mark.parametrize("n,degree,plant", [(33, 6.0, 20), (600, 10.0, 33), (3001, 12.0, 0), (5000, 14.0, 70)])
def test_against_the_oracle(ctx, n, degree, plant, k):
    if k >= 5:
        degree, plant = degree / 2, min(plant, 34)
    scale = (n - 1).bit_length()
    off, adj = cds.gen_rmat(scale, degree / 2 * n / (1 << scale), n + k, n=n)
    if plant:
        off, adj, _ = cds.gen_plant(off, adj, plant, 0.6, n)
    # a hub whose row is a block's work, joined to every third vertex
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    hub = np.arange(1, n, 3)
    off, adj = cds.csr_from_edges(n, np.r_[src, np.zeros_like(hub)], np.r_[adj.astype(np.int64), hub])
    want = oracle.peel(off, adj, k)
    g = ctx.graph(off, adj)
    core, largest, total = ctx.clique_core(g, k)
    g.free()
    assert total == want["total"]
    assert np.array_equal(core.astype(np.int64), want["core"])
    assert largest == want["core"].max()


@pytest.mark.parametrize("k,groups,m", [(3, 2100, 70), (4, 1000, 20), (5, 300, 12), (6, 200, 10)])
def test_later_sets_past_one_team(ctx, k, groups, m):
    # `groups` complete graphs of k-1 vertices, all joined to a complete graph D of
    # m; a hub joined to every group but not to D lies in one k-clique a group
    r = k - 1
    u, v = [], []

    def edge(a, b):
        u.append(a)
        v.append(b)

    first = 1 + m
    for a in range(m):
        for b in range(a):
            edge(1 + a, 1 + b)
    for gi in range(groups):
        base = first + gi * r
        for x in range(r):
            edge(0, base + x)
            for y in range(x):
                edge(base + x, base + y)
            for d in range(m):
                edge(base + x, 1 + d)
    n = first + groups * r
    off, adj = cds.csr_from_edges(n, u, v)
    # k-cliques of a group's vertex with the rest of its group and D, without the hub
    deg = sum(comb(r - 1, i) * comb(m, k - 1 - i) for i in range(r))
    assert deg > groups and comb(m - 1, k - 1) < deg
    g = ctx.graph(off, adj)
    core, largest, _ = ctx.clique_core(g, k)
    sol = ctx.solve(g, k, search="core")
    g.free()
    assert core[0] == groups
    assert (core[1:] == deg).all() and largest == deg
    assert sol.max_core == deg and sol.peel_levels == 2


@pytest.mark.parametrize("k", [3, 4])
def test_levels_of_long_histograms(ctx, k):
    # clique-core numbers on both sides of the 32,768 values from which the levels in
    # use are gathered first, alone and as one batch (whose values add up)
    graphs = []
    for m in (60, 61) if k == 4 else (256, 259):  # largest values 32,509 / 34,220; 32,385 / 33,153
        off, adj = cds.gen_er(m, 0.0, 1)
        graphs.append(cds.gen_plant(off, adj, m, 1.0, 1)[:2])
    off, adj = cds.gen_er(900, 14.0 / 900, 2)
    graphs.append(cds.gen_plant(off, adj, 90, 0.8, 3)[:2])
    graphs.append(cds.gen_er(20, 0.0, 1))  # no clique
    gs = [ctx.graph(off, adj) for off, adj in graphs]
    params = cds.make_params(k)
    batch = ctx.solve_batch([(g, params) for g in gs])
    for (off, adj), g, b in zip(graphs, gs, batch):
        s = ctx.solve(g, k)
        for r in (s, b):
            assert (r.num, r.den, r.vertices.tolist(), r.max_core, r.core_threshold) == (
                s.num, s.den, s.vertices.tolist(), s.max_core, s.core_threshold)
        g.free()
        if s.num == 0:
            continue
        if len(off) <= 260:  # a complete graph
            m = len(off) - 1
            want = np.full(m, comb(m - 1, k - 1))
        else:
            want = oracle.peel(off, adj, k)["core"]
        assert s.max_core == int(want.max())
        assert s.peel_levels == len(np.unique(want))


@pytest.mark.parametrize("gap", [0, 31, 20_000_000])
def test_long_runs_of_isolated_vertices(ctx, gap):
    # two triangles, two edges and a fan, whose arcs lie on both sides of the runs
    first = np.array([0, 0, 1, 3]), np.array([1, 2, 2, 4])
    fan = np.arange(40)
    u, v = [first[0], first[0] + 5 + gap], [first[1], first[1] + 5 + gap]
    base = 10 + 2 * gap
    u += [np.full(40, base), base + 1 + fan[:-1]]
    v += [base + 1 + fan, base + 2 + fan[:-1]]
    n = base + 41
    off, adj = cds.csr_from_edges(n, np.concatenate(u), np.concatenate(v))
    g = ctx.graph(off, adj)
    ctx.profile(True)
    ctx.profile_read()
    core, largest, total = ctx.clique_core(g, 3)
    arcs_ms = ctx.profile_read()["peel_arcs"][1]
    ctx.profile(False)
    g.free()
    want = np.zeros(n, np.int64)
    want[[0, 1, 2]] = want[np.array([0, 1, 2]) + 5 + gap] = 1
    want[base:] = 1  # a fan: every core holds a vertex of one triangle
    assert total == 2 + 39 and largest == 1
    assert np.array_equal(core.astype(np.int64), want)
    assert arcs_ms < 100  # (the runs walked one vertex after another: 3,554 ms)
