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


@pytest.mark.parametrize("n", [16380, 16385, 200005])
@pytest.mark.parametrize("more", [-2, 0])
@pytest.mark.parametrize("apart", [1, 1000])
def test_edges_a_row(sg, n, more, apart):
    """Below and at the rows and the edges a row from which later rounds follow the
    first: paths of `apart` parts, ids shuffled, and chords within the parts."""
    rng = np.random.default_rng(n + apart)
    id_ = rng.permutation(n)
    have = {(i, i + apart) for i in range(n - apart)}
    while 2 * len(have) < 16 * n // 5 + more:
        for i, k in zip(rng.integers(0, n, n).tolist(), rng.integers(1, max(n // apart, 2), n).tolist()):
            j = i + k * apart
            if j < n and 2 * len(have) < 16 * n // 5 + more:
                have.add((i, j))
    e = id_[np.array(sorted(have))]
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    e = oracle.symmetrize(e.astype(np.uint32))
    g.insert_batch(e)
    o.insert_batch(e)
    assert g.M() == 16 * n // 5 + more
    got = np.asarray(sg.CC(g))
    assert np.array_equal(got, o.cc()) and len(np.unique(got)) == apart
    g.close()
