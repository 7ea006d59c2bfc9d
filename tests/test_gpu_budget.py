"""Solves under device-memory budgets that hold them only where what speeds a stage up
(the proof by balanced shares, the bitmap of heavy vertices) gives way."""
import numpy as np
import pytest

import cds_b200 as cds

pytestmark = pytest.mark.gpu


def test_flows_where_the_proof_does_not_fit():
    # 1,000 triangles in a ring: their own densest set, and small networks
    n = 1000
    i = np.arange(n)
    off, adj = cds.csr_from_edges(n, np.r_[i, i], np.r_[(i + 1) % n, (i + 2) % n])
    with cds.Context(0) as c:
        g = c.graph(off, adj)
        want = c.solve(g, 3)
        peak = c.mem_usage()[1]
        g.free()
    assert (want.num, want.den, want.total_cliques) == (n, n, n)
    for less in (64 << 10, 96 << 10, 128 << 10):  # (the proof's arrays take about 400 KB)
        with cds.Context(0, mem_budget=peak - less) as c:
            g = c.graph(off, adj)
            got = c.solve(g, 3)
            g.free()
        assert (got.num, got.den) == (n, n)
        assert np.array_equal(got.vertices, want.vertices)


@pytest.mark.parametrize("mb", [4, 6, 33, 34, 36])
def test_bitmap_leaves_memory_to_the_stages(mb):
    # all 16,384 vertices could be heavy: a bitmap of 32 MB beside 4 MB of everything else
    off, adj = cds.gen_er(16384, 4 / 16384, 1)
    with cds.Context(0) as c:
        g = c.graph(off, adj)
        want, (wcore, *wrest) = c.solve(g, 3), c.clique_core(g, 3)
        g.free()
    with cds.Context(0, mem_budget=mb << 20) as c:
        g = c.graph(off, adj)
        got, (core, *rest) = c.solve(g, 3), c.clique_core(g, 3)
        g.free()
    assert (got.num, got.den, got.total_cliques) == (want.num, want.den, want.total_cliques)
    assert np.array_equal(got.vertices, want.vertices)
    assert np.array_equal(core, wcore) and rest == wrest
