"""Connected components at the sizes where the sampling rounds change, on
graphs of many components, against the CPU oracle (labels equal)."""
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


# a single vertex; below, at and above the size from which later rounds sample
@pytest.mark.parametrize("n", [1, 31, 1000, (1 << 17) - 1, 1 << 17, (1 << 17) + 33])
@pytest.mark.parametrize("shape", ["sparse", "path", "cliques", "er8"])
def test_components(sg, n, shape):
    rng = np.random.default_rng(n)
    if shape == "sparse":      # average degree 1: thousands of components
        e = rng.integers(0, n, (n // 2, 2))
    elif shape == "path":      # one long component, ids shuffled along it
        p = rng.permutation(n)
        e = np.stack([p[:-1], p[1:]], 1)
    elif shape == "cliques":   # components of nine vertices far apart in id
        k = max(n // 9, 1)
        e = np.concatenate([np.stack([np.arange(n - k), np.arange(k, n)], 1)]) if n > k else np.zeros((0, 2))
    else:
        e = rng.integers(0, n, (4 * n, 2))
    e = oracle.symmetrize(e.astype(np.uint32)) if len(e) else np.zeros((0, 2), np.uint32)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    if len(e):
        g.insert_batch(e)
        o.insert_batch(e)
    assert np.array_equal(sg.CC(g), o.cc())


@pytest.mark.parametrize("n,m", [(1000, 1500), (200000, 400000), (200000, 900000)])
def test_one_way_edges(sg, n, m):
    """Edges stored in one direction only: the same labels at every call, and
    those of the byte-width snapshot, whose links are single ones."""
    rng = np.random.default_rng(m)
    g = sg.SparseMatrixV(n)
    g.insert_batch(rng.integers(0, n, (m, 2)).astype(np.uint32))
    want = np.asarray(sg.CC(g))
    c = sg.CompactGraph(g)
    assert np.array_equal(np.asarray(c.cc()), want)
    for _ in range(3):
        assert np.array_equal(np.asarray(sg.CC(g)), want)
    c.close()
    g.close()
