"""Triangles, the total and by vertex, on the graph and on the byte-width
snapshot, against counts known in closed form or from the adjacency matrix:
rows of one and of many leaves, oriented lists that fit the hash set on both
ends of an edge, on one and on none, with and without stored self-loops.  (A
loop belongs to no triangle; loops once matched a vertex's list against itself.)
The count's two forms: by rows (up to 65,536 items, or where lists differ in
length, as a skewed graph's do) and by oriented lists."""
import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    import __graft_entry__ as ge
    ge.build()
    import sstgraph_gb300
    return sstgraph_gb300


def both(u, v):
    e = np.stack([u, v], 1)
    return np.concatenate([e, e[:, ::-1]]).astype(np.uint32)


def clique(k):
    u, v = np.triu_indices(k, 1)
    return both(u, v)


def random(n, m, seed):
    e = np.random.default_rng(seed).integers(0, n, (m, 2))
    e = e[e[:, 0] != e[:, 1]]
    return both(e[:, 0], e[:, 1])


def by_matrix(n, e):
    a = np.zeros((n, n))
    a[e[:, 0], e[:, 1]] = 1
    pv = ((a @ a) * a).sum(1).astype(np.int64) // 2  # exact: below 2^53
    return int(pv.sum()) // 3, pv


def check(sg, n, e, loops, total, pv):
    g = sg.SparseMatrixV(n, keep_self_loops=loops)
    g.insert_batch(e)
    if loops:
        v = np.arange(n, dtype=np.uint32)
        g.insert_batch(np.stack([v, v], 1))
        assert g.has(0, 0)
    c = sg.CompactGraph(g)
    for tc in (lambda **kw: sg.TC(g, **kw), c.tc):
        assert tc() == total
        got, by = tc(per_vertex=True)
        assert got == total
        assert np.array_equal(np.asarray(by).astype(np.int64), pv)
    c.close()
    g.close()


# lists of one entry; one leaf; many leaves; the longest above the 1024 entries
# of a set, on both ends of an edge among the lowest 176 vertices
@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("k", [3, 20, 33, 300, 1200])
def test_clique(sg, k, loops):
    check(sg, k, clique(k), loops, math.comb(k, 3), np.full(k, math.comb(k - 1, 2)))


@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("n,m", [(50, 100), (300, 3000), (1500, 100000), (2000, 2500)])
def test_random(sg, n, m, loops):
    e = random(n, m, n)
    check(sg, n, e, loops, *by_matrix(n, e))


# items below and above the 65,536 that are counted by rows unseen; uniform graphs
# (by lists) and skewed ones (by rows); a path and a star, whose lists hold one entry
@pytest.mark.parametrize("loops", [False, True])
@pytest.mark.parametrize("shape", ["er16000", "er16400", "er40000", "rmat14", "rmat16", "path", "star",
                                   "er65500", "er65600", "er90000", "rmat17", "path90000", "star90000"])
def test_forms(sg, shape, loops):
    rng = np.random.default_rng(5)
    if shape[:4] == "path":
        n = int(shape[4:] or 30000)
        e = both(np.arange(n - 1), np.arange(1, n))
    elif shape[:4] == "star":
        n = int(shape[4:] or 30000)
        e = np.concatenate([both(np.full(n - 1, 7), np.setdiff1d(np.arange(n), [7])), both([1], [2])])
    elif shape[:2] == "er":
        n = int(shape[2:])
        e = rng.integers(0, n, (8 * n, 2))
        e = both(*e[e[:, 0] != e[:, 1]].T)
    else:
        n = 1 << int(shape[4:])
        e = oracle.symmetrize(oracle.rmat(int(shape[4:]), 8 * n, seed=4))
        e = e[e[:, 0] != e[:, 1]]
    o = oracle.OracleGraph(n)
    o.insert_batch(e)
    total, pv = o.tc(per_vertex=True)
    check(sg, n, e, loops, total, np.asarray(pv).astype(np.int64))
