"""Core numbers past the oracle's reach, checked by deletion: {core >= L} has to be what
is left of the graph when vertices in fewer than L cliques are deleted until there is
none.  The clique degrees on the way come from the counting of each induced graph,
which shares neither order nor sweeps with the core numbers."""
import numpy as np
import pytest

import cds_b200 as cds

pytestmark = pytest.mark.gpu


def induced(off, adj, keep):
    src = np.repeat(np.arange(len(off) - 1), np.diff(off.astype(np.int64)))
    on = keep[src] & keep[adj]
    ids = np.cumsum(keep) - 1
    new = np.zeros(int(keep.sum()) + 1, np.uint64)
    new[1:] = np.cumsum(np.bincount(ids[src[on]], minlength=len(new) - 1))
    return new, ids[adj[on]].astype(np.uint32)


def left_by_deletion(ctx, off, adj, degree, k, level):
    ids = np.arange(len(off) - 1)
    while True:
        keep = degree >= level
        ids = ids[keep]
        if keep.all() or not len(ids):
            return ids
        off, adj = induced(off, adj, keep)
        g = ctx.graph(off, adj)
        degree = ctx.list_cliques(g, k)[1]
        g.free()


@pytest.mark.parametrize("scale,factor,plant,k", [(16, 12, 0, 3), (16, 12, 0, 4), (15, 6, 60, 5), (13, 6, 0, 6),
                                                 (18, 16, 300, 4)])
def test_levels_by_deletion(scale, factor, plant, k):
    off, adj = cds.gen_rmat(scale, factor, 4)
    if plant:
        off, adj, _ = cds.gen_plant(off, adj, plant, 0.5, 4)
    with cds.Context(0) as ctx:
        g = ctx.graph(off, adj)
        core = ctx.clique_core(g, k)[0].astype(np.int64)
        degree = ctx.list_cliques(g, k)[1]
        g.free()
        values = np.unique(core[core > 0])
        for level in {1, int(values[len(values) // 2]), int(values[-1 - len(values) // 20]), int(values[-1])}:
            want = np.flatnonzero(core >= level)
            assert np.array_equal(left_by_deletion(ctx, off, adj, degree, k, level), want)
        # (no core above the largest)
        assert not len(left_by_deletion(ctx, off, adj, degree, k, int(values[-1]) + 1))


def hubs_over_blocks(blocks, seed):
    """Random blocks of 24 vertices, denser and sparser ones; hubs joined to a few vertices
    of each block, whose values lie among the blocks'; beside them 620 vertices of degree
    about 590, so many rows of over 512 entries that warps order rows of up to 2,048."""
    rng = np.random.default_rng(seed)
    u, v = [], []
    x, y = np.triu_indices(24, 1)
    for b in range(blocks):
        on = rng.random(len(x)) < rng.uniform(0.8, 1.0)
        u.append(x[on] + 24 * b)
        v.append(y[on] + 24 * b)
    n = 24 * blocks
    for _ in range(6):
        near = np.concatenate([24 * b + rng.choice(24, rng.integers(3, 5), replace=False) for b in range(blocks)])
        u.append(np.full(len(near), n))
        v.append(near)
        n += 1
    x, y = np.triu_indices(620, 1)
    on = rng.random(len(x)) < 0.95
    u.append(x[on] + n)
    v.append(y[on] + n)
    return cds.csr_from_edges(n + 620, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("blocks,k", [(260, 4), (300, 4), (380, 4), (300, 3)])
def test_many_wide_rows_with_later_sets_past_one_team(blocks, k):
    # hubs' later sets past the 768 vertices that one block counts, recounted as the
    # blocks' values fall below the hubs'
    off, adj = hubs_over_blocks(blocks, blocks)
    with cds.Context(0) as ctx:
        g = ctx.graph(off, adj)
        core = ctx.clique_core(g, k)[0].astype(np.int64)
        degree = ctx.list_cliques(g, k)[1]
        g.free()
        values = np.unique(np.r_[core[24 * blocks:24 * blocks + 6], np.unique(core)[[1, -1]]])
        for level in np.unique(np.r_[values, values + 1]):
            want = np.flatnonzero(core >= level)
            assert np.array_equal(left_by_deletion(ctx, off, adj, degree, k, level), want)
