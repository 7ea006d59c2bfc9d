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
