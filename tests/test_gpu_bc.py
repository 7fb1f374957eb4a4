"""Single-source dependencies, against the CPU oracle: rows of one leaf, of each
capacity class up to 32 leaves and hubs of several chunks, in levels that are pushed
(queued) and pulled (found in the lists), at every mix of the two and with chunks of
one leaf and of 32; and the search's depths beside them."""
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


def layered(rng):
    """a source, then layers of hubs of 2 .. 64 leaves and their ends, each end in
    a row of the next layer: queued and unqueued levels of every class"""
    e, v, last = [], 1, np.array([0])
    for k in (40, 90, 200, 500, 900, 1500, 3000):
        hubs = np.arange(v, v + 4)
        ends = np.arange(v + 4, v + 4 + k)
        v += 4 + k
        e += [np.stack(np.meshgrid(last[:50], hubs), -1).reshape(-1, 2)]
        e += [np.stack(np.meshgrid(hubs, ends), -1).reshape(-1, 2)]
        last = ends
    return v, np.concatenate(e)


def shapes():
    rng = np.random.default_rng(8)
    yield "pair", 2, np.array([[0, 1]])
    yield "path", 700, np.stack([np.arange(699), np.arange(1, 700)], 1)
    n, e = layered(rng)
    yield "layers", n, e
    yield "er", 20000, rng.integers(0, 20000, (60000, 2))
    yield "rmat", 1 << 14, oracle.rmat(14, 10 << 14, seed=5)
    yield "dense", 600, rng.integers(0, 600, (50000, 2))


@pytest.fixture(scope="module", params=[s[0] for s in shapes()])
def pair(request, sg):
    name, n, e = next(s for s in shapes() if s[0] == request.param)
    e = e[e[:, 0] != e[:, 1]]
    e = oracle.symmetrize(e.astype(np.uint32))
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    g.insert_batch(e)
    o.insert_batch(e)
    return g, o


# alpha 1: push unless the frontier holds all edges; 1 << 30: pull from the start
@pytest.mark.parametrize("alpha", [1, 20, 1 << 30])
@pytest.mark.parametrize("chunk", [1, 8, 32])
def test_dependencies(sg, pair, alpha, chunk):
    g, o = pair
    sg.set_tuning(g, chunk_leaves=chunk, bfs_alpha=alpha)
    for src in sorted({0, g.rows // 2, g.rows - 1}):
        got, want = np.asarray(sg.BC(g, src)), o.bc(src)
        # positive sums: below 2^12 terms a vertex, a product and a quotient, over
        # below 2^10 levels, each rounded once
        assert np.all(np.abs(got - want) <= 2.0 ** -53 * 2 ** 23 * want)
        assert np.array_equal(sg.BFS(g, src, depths=True), o.bfs(src))


def test_same_sums_at_every_mix(sg, pair):
    """a vertex's sum is added up in one order, whichever way its level was reached"""
    g, o = pair
    sg.set_tuning(g, chunk_leaves=32, bfs_alpha=20)
    want = np.asarray(sg.BC(g, 0)).copy()
    for alpha in (1, 3, 1 << 30):
        sg.set_tuning(g, chunk_leaves=32, bfs_alpha=alpha)
        assert np.array_equal(np.asarray(sg.BC(g, 0)), want)
