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
