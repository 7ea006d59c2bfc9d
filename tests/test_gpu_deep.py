"""Clique sizes past 5 on neighbourhoods of several words: totals, clique degrees and
clique-core numbers against the oracle where the search over common neighbours
changes its way -- rows of one word, of two to four, wider ones; depths with and
without a search of their own (k = 6, 7 and more).  Exact."""
import numpy as np
import pytest

import cds_b200 as cds
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with cds.Context(0) as c:
        yield c


def graph(n, p, plants, seed):
    """A random graph with complete subgraphs that overlap it at random."""
    rng = np.random.default_rng(seed)
    x, y = np.triu_indices(n, 1)
    on = rng.random(len(x)) < p
    for size in plants:
        inside = np.zeros(n, bool)
        inside[rng.choice(n, size, replace=False)] = True
        on |= inside[x] & inside[y]
    return cds.csr_from_edges(n, x[on], y[on])


# later neighbourhoods of up to about n p vertices
SHAPES = [(40, 0.7, ()), (90, 0.5, (12,)), (150, 0.4, (14, 9)), (320, 0.36, (13,)), (700, 0.23, (15, 11))]


@pytest.mark.parametrize("k", [6, 7, 8, 9, 12])
@pytest.mark.parametrize("n,p,plants", SHAPES)
def test_against_the_oracle(ctx, n, p, plants, k):
    off, adj = graph(n, p if k < 9 else p * 0.7, plants, n + k)
    g = ctx.graph(off, adj)
    count, degree = ctx.list_cliques(g, k)
    core, largest, total = ctx.clique_core(g, k)
    g.free()
    want, wdeg = oracle.count_cliques(off, adj, k)
    assert count == total == want
    assert np.array_equal(degree.astype(np.int64), np.asarray(wdeg, np.int64))
    assert np.array_equal(core.astype(np.int64), oracle.peel(off, adj, k)["core"])
