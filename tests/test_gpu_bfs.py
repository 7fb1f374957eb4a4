"""Breadth-first search with every mix of push and pull levels, on graphs whose
rows and levels have the sizes where its work splits change, against the CPU
oracle (depths equal; a parent is a neighbour one level up)."""
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


def stars(n, rng):
    """hubs of 1, 2, 4, 5, 33 and more leaves, each hub next to the next one"""
    e, v = [], 8
    for h, k in enumerate((20, 33, 60, 65, 130, 161, 1100, 3000)):
        ends = np.arange(v, v + k)
        v += k
        e += [np.stack([np.full(k, h), ends], 1)]
        if h:
            e += [np.array([[h - 1, h]])]
    return np.concatenate(e)


def shapes():
    rng = np.random.default_rng(2)
    yield "one", 1, np.zeros((0, 2))
    yield "pair", 2, np.array([[0, 1]])
    yield "path", 1500, np.stack([np.arange(1499), np.arange(1, 1500)], 1)
    yield "stars", 6000, stars(6000, rng)
    yield "er", 33333, rng.integers(0, 33333, (100000, 2))
    yield "rmat", 1 << 15, oracle.rmat(15, 10 << 15, seed=3)
    yield "dense", 700, rng.integers(0, 700, (60000, 2))


@pytest.fixture(scope="module", params=[s[0] for s in shapes()])
def pair(request, sg):
    name, n, e = next(s for s in shapes() if s[0] == request.param)
    e = oracle.symmetrize(e.astype(np.uint32)) if len(e) else np.zeros((0, 2), np.uint32)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    if len(e):
        g.insert_batch(e)
        o.insert_batch(e)
    return g, o


# alpha 1: push unless the frontier holds all edges; 20: the default mix;
# 1 << 30: pull from the first level on.  Leaf chunks of 32, 8 and 1
@pytest.mark.parametrize("alpha,chunk", [(1, 32), (3, 8), (20, 32), (1 << 30, 32), (1 << 30, 1)])
def test_levels(sg, pair, alpha, chunk):
    g, o = pair
    sg.set_tuning(g, chunk_leaves=chunk, bfs_alpha=alpha)
    off, cols = o.csr()
    for src in sorted({0, g.rows // 2, g.rows - 1}):
        want = o.bfs(src)
        par, dep = sg.BFS_both(g, src)
        assert np.array_equal(dep, want)
        assert np.array_equal(sg.BFS(g, src, depths=True), want)
        assert par[src] == src and np.all(par[want < 0] == -1)
        v = np.nonzero(want > 0)[0]
        assert np.array_equal(want[par[v]], want[v] - 1)
        for x in v[:: max(1, len(v) // 300)]:
            assert par[x] in cols[off[x]:off[x + 1]]
