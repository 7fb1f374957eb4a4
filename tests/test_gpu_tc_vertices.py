"""Triangles at listed vertices: few and many of them (chunks of 2, 4, 8 and 32
leaves), rows of one and of many leaves, against the oracle and, on larger
graphs, the count over all vertices."""
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


@pytest.mark.parametrize("k", [1, 7, 300, 2000])
def test_few_vertices(sg, k):
    n = 2000
    rng = np.random.default_rng(k)
    e = rng.integers(0, n, (6000, 2)).astype(np.uint32)
    c = np.stack(np.meshgrid(np.arange(150), np.arange(150)), -1).reshape(-1, 2).astype(np.uint32)
    hub = np.stack([np.zeros(n, np.uint32), np.arange(n, dtype=np.uint32)], 1)
    e = oracle.symmetrize(np.concatenate([e, c, hub]))  # one-leaf rows, a clique, a hub
    g = sg.SparseMatrixV(n)
    g.insert_batch(e)
    o = oracle.OracleGraph(n)
    o.insert_batch(e)
    _, pv = o.tc(per_vertex=True)
    vs = rng.permutation(n)[:k].astype(np.uint32)
    vs[0] = 0
    assert np.array_equal(sg.TC_vertices(g, vs), np.asarray(pv)[vs])
    g.close()


@pytest.mark.parametrize("scale", [13, 15, 17])
def test_all_vertices(sg, scale):
    n = 1 << scale
    g = sg.SparseMatrixV(n)
    g.insert_batch(oracle.symmetrize(oracle.rmat(scale, 8 * n, seed=scale)))
    vs = np.arange(n, dtype=np.uint32)
    _, pv = sg.TC(g, per_vertex=True)
    assert np.array_equal(sg.TC_vertices(g, vs), np.asarray(pv))
    g.close()
