"""A sequential model of the clique-core numbers by arc weights (k_core in
cds_b200/csrc/peel.cu), checked against the oracle's peel on small graphs.

The model keeps the kernel's rules and randomises what the GPU leaves to scheduling:
  * an order by value; ties keep the order they had, a vertex that arrives at a value
    goes behind those that were there;
  * a sweep recounts the weights of the roots whose later set changed, and only of
    vertices within the range of the changes since the last order;
  * then lowers, `lower` times at most, every vertex within the range of the changes since,
    in a random order and at once: the weighted h-index over weights that
    get older from one pass to the next;
  * a first pass (weights current) that lowers nothing ends it.
No value may fall below the core number, a vertex outside the range may have nothing to
lower and no other later set, and the last values are the core numbers."""
import random
from itertools import combinations

import numpy as np
import pytest

import cds_b200 as cds
import oracle


def h_index(rooted, weights, tau, limit):
    """The largest h <= limit with at least h cliques: `rooted` count for every h, weight
    c of an earlier root u where tau(u) >= h."""
    h = limit
    while h and rooted + sum(c for u, c in weights.items() if tau[u] >= h) < h:
        h -= 1
    return h


def core_numbers(off, adj, k, lower, rng, want):
    n = len(off) - 1
    near = [set(adj[int(off[v]):int(off[v + 1])].tolist()) for v in range(n)]

    def cliques(inside, size):  # of a set, as tuples
        return [c for c in combinations(sorted(inside), size)
                if all(b in near[a] for a, b in combinations(c, 2))]

    tau = np.asarray(oracle.count_cliques(off, adj, k)[1], np.int64).tolist()
    arrival = [0] * n  # sweep a vertex arrived at its value in
    fell = [0] * n     # and how far it fell then
    seen = list(tau)   # value when last ordered
    later = [None] * n
    rooted, weights = [0] * n, [{} for _ in range(n)]
    reach = (0, 1 << 60)
    for sweep in range(10000):
        for v in range(n):
            if tau[v] != seen[v]:
                arrival[v], fell[v], seen[v] = sweep, seen[v] - tau[v], tau[v]
        key = [(tau[v], arrival[v], fell[v], v) for v in range(n)]
        for u in range(n):
            if not tau[u]:
                continue
            now = {w for w in near[u] if key[w] > key[u]}
            if not reach[0] <= tau[u] <= reach[1]:
                assert now == later[u]
                continue
            if now == later[u]:
                continue
            for w in (later[u] or set()) | now:
                weights[w].pop(u, None)
            later[u] = now
            found = cliques(now, k - 1)
            rooted[u] = len(found)
            for c in found:
                for w in c:
                    weights[w][u] = weights[w].get(u, 0) + 1
        moved = None
        for x in range(lower):
            low, high = 1 << 60, -1
            for v in rng.sample(range(n), n):
                if not tau[v]:
                    continue
                h = h_index(rooted[v], weights[v], tau, tau[v])
                assert h >= want[v]
                if not reach[0] <= tau[v] <= reach[1]:
                    # looked at next where a change of this pass reaches it
                    assert h == tau[v] or low <= tau[v] <= high
                elif h < tau[v]:
                    low, high = min(low, h), max(high, tau[v])
                    tau[v] = h
            reach = (low, high)
            if high >= 0:
                moved = (low, high) if moved is None else (min(low, moved[0]), max(high, moved[1]))
            else:
                if x == 0:
                    return tau
                break
        reach = moved
    raise AssertionError("no fixpoint")


@pytest.mark.parametrize("k", [3, 4, 5])
@pytest.mark.parametrize("lower", [1, 2, 4])
@pytest.mark.parametrize("seed", range(4))
def test_model_reaches_the_core_numbers(k, lower, seed):
    n = 40 + 7 * seed
    off, adj = cds.gen_er(n, 0.25 if seed % 2 else 0.12, seed + 11 * k)
    off, adj, _ = cds.gen_plant(off, adj, 12 + seed, 0.8, seed)
    want = oracle.peel(off, adj, k)["core"].tolist()
    assert core_numbers(off, adj, k, lower, random.Random(seed * 31 + lower), want) == want


@pytest.mark.parametrize("lower", [1, 2])
def test_model_on_a_chain(lower):
    # a strip of triangles: changes come in from both ends, a vertex or two a sweep
    n = 30
    i = np.arange(n)
    off, adj = cds.csr_from_edges(n, np.r_[i[:-1], i[:-2]], np.r_[i[1:], i[2:]])
    want = oracle.peel(off, adj, 3)["core"].tolist()
    assert core_numbers(off, adj, 3, lower, random.Random(lower), want) == want
