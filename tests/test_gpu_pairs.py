"""Pairwise queries at the edges of their kernels' work splits, against the
CPU oracle (whole numbers: equal)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

N = 6000


@pytest.fixture(scope="module")
def sg():
    import __graft_entry__ as ge
    ge.build()
    import sstgraph_gb300
    return sstgraph_gb300


@pytest.fixture(scope="module")
def graph(sg):
    """Rows of every shape: hubs of many leaves, rows of one leaf at each
    capacity, empty rows."""
    rng = np.random.default_rng(3)
    hubs = [np.stack([np.full(k, v), rng.choice(N, k, replace=False)], 1)
            for v, k in ((0, 5900), (1, 3000), (2, 700), (3, 65))]
    rest = [np.stack([np.full(k, 10 + k), rng.choice(N, k, replace=False)], 1)
            for k in range(1, 41)]
    noise = rng.integers(100, N - 100, (20000, 2))
    edges = oracle.symmetrize(np.concatenate(hubs + rest + [noise]).astype(np.uint32))
    g, o = sg.SparseMatrixV(N), oracle.OracleGraph(N)
    g.insert_batch(edges)
    o.insert_batch(edges)
    return g, o


def pairs_of(n):
    rng = np.random.default_rng(n)
    p = rng.integers(0, N, (n, 2)).astype(np.uint32)
    hub = rng.random((n, 2)) < 0.3
    p[hub] = rng.integers(0, 55, int(hub.sum()))
    return p


# 1 pair; a block's share and one more; the clusters' shares (2 blocks an SM,
# 64 pairs a block at most) filled unevenly
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 303, 305, 513, 4099, 20011])
@pytest.mark.parametrize("early", [False, True])
def test_common_neighbors(graph, n, early):
    g, o = graph
    p = pairs_of(n)
    if n > 4:
        p[1] = (0, 1)    # two hubs
        p[2] = (7, 7)    # a row with itself
        p[3] = (N, 1)    # an id out of range
        p[4] = (N - 1, 0)
    got = g.common_neighbors_batch(p, early)
    exp = [0 if max(a, b) >= N else o.common_neighbors(int(a), int(b), early) for a, b in p]
    assert np.array_equal(got, np.array(exp, np.uint64))


# blocks of 64 pairs, of two and a half rounds, of as many as they hold (512)
@pytest.mark.parametrize("n", [48640, 48641, 100003, 389121])
def test_common_neighbors_of_many(graph, n):
    g, o = graph
    p = pairs_of(n)
    off, cols = o.csr()
    a = np.zeros((N, N), bool)
    a[np.repeat(np.arange(N), np.diff(off.astype(np.int64))), cols] = True
    bits = np.packbits(a, axis=1)
    ones = np.unpackbits(np.arange(256, dtype=np.uint8)[:, None], axis=1).sum(1).astype(np.uint16)
    got = np.asarray(g.common_neighbors_batch(p))
    for i in range(0, n, 20000):
        both = bits[p[i:i + 20000, 0]] & bits[p[i:i + 20000, 1]]
        assert np.array_equal(got[i:i + 20000], ones[both].sum(1))


@pytest.mark.parametrize("n", [1, 255, 256, 257, 20011])
def test_has_batch(graph, n):
    """Lookups in rows of every capacity, at and beside the ids they hold."""
    g, o = graph
    p = pairs_of(n)
    off, cols = o.csr()
    rng = np.random.default_rng(n + 1)
    for i in range(0, n, 2):  # an id of the row, or the one before or after it
        u = p[i, 0]
        if off[u + 1] > off[u]:
            x = int(cols[rng.integers(off[u], off[u + 1])]) + int(rng.integers(-1, 2))
            p[i, 1] = min(max(x, 0), N - 1)
    if n > 4:
        p[1] = (0, 0xFFFFFFFF)  # the gap marker is no id
        p[2] = (50, 0xFFFFFFFF)
        p[3] = (N, 1)
    exp = [p[i, 0] < N and p[i, 1] < N and o.has(int(p[i, 0]), int(p[i, 1])) for i in range(n)]
    assert np.array_equal(g.has_batch(p), np.array(exp, np.uint8))
