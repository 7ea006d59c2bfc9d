"""Clique counting on local bitmaps: totals and clique degrees against the
oracle (or the closed form of complete graphs) where the row building changes
its way -- graphs around the size up to which every vertex is heavy, mixed heavy
and light neighbourhoods, none heavy for lack of memory, neighbourhoods around
one word, several words and the shared-memory limit.  Counts are exact."""
from math import comb

import numpy as np
import pytest

import cds_b200 as cds
import oracle

pytestmark = pytest.mark.gpu


def complete(sizes):
    """Disjoint complete graphs."""
    off, adj, base = [0], [], 0
    for s in sizes:
        for v in range(s):
            adj.extend(base + w for w in range(s) if w != v)
            off.append(len(adj))
        base += s
    return np.array(off, np.uint64), np.array(adj, np.uint32)


@pytest.fixture(scope="module")
def ctx():
    with cds.Context(0) as c:
        yield c


def check(c, off, adj, k):
    want, deg = oracle.count_cliques(off, adj, k)
    g = c.graph(off, adj)
    got, gdeg = c.list_cliques(g, k)
    g.free()
    assert got == want
    assert np.array_equal(gdeg.astype(np.int64), np.asarray(deg, np.int64))


@pytest.mark.parametrize("k", [3, 4, 5, 6, 7])
@pytest.mark.parametrize("n", [16383, 16385, 40001])
def test_heavy_and_light(ctx, n, k):
    off, adj = cds.gen_rmat((n - 1).bit_length(), 3.0 * n / (1 << (n - 1).bit_length()), n + k, n=n)
    off, adj, _ = cds.gen_plant(off, adj, 60 if k < 6 else 45, 0.6, n)
    check(ctx, off, adj, k)


@pytest.mark.parametrize("k", [3, 4, 5, 6])
def test_no_memory_for_the_bitmap(k):
    # the whole bitmap of 9,001 vertices takes 10 MB: fewer heavy vertices fit
    off, adj = cds.gen_rmat(14, 8.0 * 9001 / 16384, 5, n=9001)
    with cds.Context(0, mem_budget=5 << 20) as small:
        check(small, off, adj, k)


@pytest.mark.parametrize("sizes", [(2, 3, 4, 5), (32, 33, 34), (64, 65, 66, 97), (128, 129, 130, 131)])
@pytest.mark.parametrize("k", [3, 4, 5, 6])
def test_neighbourhood_sizes(ctx, sizes, k):
    off, adj = complete(sizes)
    g = ctx.graph(off, adj)
    got, deg = ctx.list_cliques(g, k)
    g.free()
    assert got == sum(comb(s, k) for s in sizes)
    assert deg.tolist() == [comb(s - 1, k - 1) for s in sizes for _ in range(s)]


@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("s", [1025, 1026, 1100])
def test_rows_past_shared_memory(ctx, s, k):
    off, adj = complete((s, 40))
    g = ctx.graph(off, adj)
    got, deg = ctx.list_cliques(g, k)
    g.free()
    assert got == comb(s, k) + comb(40, k)
    assert deg.tolist() == [comb(s - 1, k - 1)] * s + [comb(39, k - 1)] * 40


# Cliques are also written where the rows are in global memory: sizes on both sides of
# a multiple of 32 and where either pass has the wider rows.  All are past the proof's
# component size, so the core's cliques are listed for the flows.
@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("s", [1026, 1122, 1140, 1152, 1398])
def test_rows_past_shared_memory_are_written(ctx, s, k):
    # s vertices joined to s others, which form s / (k-1) cliques among themselves
    r = k - 1
    low, high = np.meshgrid(np.arange(s), np.arange(s, 2 * s))
    group = np.arange(s, 2 * s).reshape(-1, r)
    x, y = np.triu_indices(r, 1)
    off, adj = cds.csr_from_edges(2 * s, np.r_[low.ravel(), group[:, x].ravel()],
                                  np.r_[high.ravel(), group[:, y].ravel()])
    g = ctx.graph(off, adj)
    sol = ctx.solve(g, k)
    g.free()
    # x low vertices and y groups hold x y cliques: most of them a vertex for all
    assert sol.total_cliques == s * (s // r) == sol.num
    assert sol.den == 2 * s and sol.vertices.tolist() == list(range(2 * s))


@pytest.mark.parametrize("s", [1122, 1140, 1153, 1400])
def test_complete_graphs_past_the_proof(ctx, s):
    off = np.arange(s + 1, dtype=np.uint64) * (s - 1)
    adj = np.broadcast_to(np.arange(s, dtype=np.uint32), (s, s))[~np.eye(s, dtype=bool)]
    g = ctx.graph(off, adj)
    sol = ctx.solve(g, 3)
    g.free()
    assert (sol.total_cliques, sol.num, sol.den) == (comb(s, 3), comb(s, 3), s)
    assert sol.vertices.tolist() == list(range(s))


@pytest.mark.parametrize("k", [6, 7, 8, 12, 16])
def test_one_word_neighbourhoods_of_large_cliques(ctx, k):
    sizes = (k - 1, k, k + 1, 20) + ((32, 33) if k < 12 else (24,))
    off, adj = complete(sizes)
    g = ctx.graph(off, adj)
    got, deg = ctx.list_cliques(g, k)
    core, _, _ = ctx.clique_core(g, k)
    g.free()
    assert got == sum(comb(s, k) for s in sizes)
    assert deg.tolist() == [comb(s - 1, k - 1) for s in sizes for _ in range(s)] == core.tolist()
    off, adj = cds.gen_er(300, 0.0, 1)
    for i in range(3):
        off, adj, _ = cds.gen_plant(off, adj, 30, 0.8 if k < 12 else 0.95, 10 * k + i)
    check(ctx, off, adj, k)
