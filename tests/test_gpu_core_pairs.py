"""Pruning and components of a small core for k >= 6, where the listed cliques mark
their pairs: cliques whose arcs climb in degree towards smaller ids, on cores of one bitmap word
and of more, against closed forms and the oracle."""
from math import comb

import numpy as np
import pytest

import cds_b200 as cds
import oracle

pytestmark = pytest.mark.gpu


def falling(blocks, base=0):
    """Complete graphs on consecutive ids (sizes `blocks`, each sharing `base` ids with
    the one before), with pendant vertices so that degrees fall with the id."""
    u, v, first = [], [], 0
    for s in blocks:
        x, y = np.triu_indices(s, 1)
        u.append(x + first)
        v.append(y + first)
        first += s - base
    n = first + base
    extra = np.concatenate([np.full(n - i, i) for i in range(n)])  # more than any difference in blocks
    leaf = n + np.arange(len(extra))
    return cds.csr_from_edges(n + len(extra), np.r_[np.concatenate(u), extra], np.r_[np.concatenate(v), leaf])


def answer(off, adj, k):
    with cds.Context(0) as c:
        g = c.graph(off, adj)
        s = c.solve(g, k)
        got = c.components(g, k)
        g.free()
    assert (s.n_components, s.pruned_edges) == (len(got["components"]), got["pruned_edges"])
    return s


# (blocks, vertices shared; vertices of the answer, components of the core): a smaller
# block beside larger ones is below the core's threshold
@pytest.mark.parametrize("k", [6, 7])
@pytest.mark.parametrize("blocks,shared,size,parts", [((20,), 0, 20, 1), ((32,), 0, 32, 1), ((33,), 0, 33, 1),
                                                      ((40,), 0, 40, 1), ((36, 36), 0, 36, 2), ((36, 36), 8, 64, 1),
                                                      ((40, 12, 40), 0, 40, 2)])
def test_arcs_towards_smaller_ids(blocks, shared, size, parts, k):
    off, adj = falling(blocks, shared)
    s = answer(off, adj, k)
    top, copies = max(blocks), 2 if shared else 1
    assert (s.num, s.den) == (copies * comb(top, k) - (copies - 1) * comb(shared, k), size)
    assert s.vertices.tolist() == list(range(size))
    assert s.n_components == parts
    assert s.pruned_edges == blocks.count(top) * comb(top, 2) - comb(shared, 2)


@pytest.mark.parametrize("k", [6, 7])
def test_random_core(k):
    off, adj = cds.gen_er(46, 0.0, 1)
    off, adj, _ = cds.gen_plant(off, adj, 46, 0.55, k)
    n = len(off) - 1
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    extra = np.concatenate([np.full(2 * (n - i), i) for i in range(n)])
    off, adj = cds.csr_from_edges(n + len(extra), np.r_[src, extra],
                                  np.r_[adj.astype(np.int64), n + np.arange(len(extra))])
    want = oracle.solve(off, adj, k)
    s = answer(off, adj, k)
    assert (s.num, s.den, s.n_components, s.pruned_edges) == tuple(
        want[x] for x in ("num", "den", "n_components", "pruned_edges"))
    assert s.vertices.tolist() == want["vertices"].tolist()
