"""Searches of graphs most of whose vertices have no edge: the arrays of all
vertices are cleared and read whatever the rows in use, and where those are few
(below an eighth) BC clears theirs alone and (below a half) components pass over
them alone.  Against the CPU oracle, before and after updates that take the graph
past those shares and back."""
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


def compare(sg, g, o, srcs):
    for src in srcs:
        assert np.array_equal(sg.BFS(g, src, depths=True), o.bfs(src))
        got, want = np.asarray(sg.BC(g, src)), o.bc(src)
        # sums of below 2^16 positive terms a vertex over below 2^4 levels, in FP64
        assert np.all(np.abs(got - want) <= 2.0 ** -53 * 2 ** 20 * np.maximum(np.abs(want), 1e-300))
    assert np.array_equal(sg.CC(g), o.cc())


# rows in use of all: none, one edge, one in 40, below and above an eighth and a half
@pytest.mark.parametrize("n", [4096, (1 << 17) - 1, (1 << 18) + 7])
@pytest.mark.parametrize("share", [0, 2, 40, 9, 7, 1.9, 1.1])
def test_share_in_use(sg, n, share):
    rng = np.random.default_rng(n + int(10 * share))
    used = rng.permutation(n)[: (0 if share == 0 else 2 if share == 2 else int(n / share))]
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    idle = int(np.setdiff1d(np.arange(n), used)[0])

    def step(op, e):
        e = oracle.symmetrize(e.astype(np.uint32))
        for m in (g, o):
            getattr(m, op)(e)

    if len(used):
        e = used[rng.integers(0, len(used), (4 * len(used), 2))]
        hub = np.stack([np.full(min(len(used), 3000), used[0]), used[:3000]], 1)
        e = np.concatenate([e, hub])
        e = e[e[:, 0] != e[:, 1]]
        if len(e):
            step("insert_batch", e)
    srcs = [idle] + ([int(used[0]), int(used[-1])] if len(used) else [])
    compare(sg, g, o, srcs)
    more = rng.integers(0, n, (n // 4, 2))
    more = more[more[:, 0] != more[:, 1]]
    step("insert_batch", more)
    compare(sg, g, o, srcs[:2])
    step("remove_batch", more)
    compare(sg, g, o, srcs)
    g.close()


@pytest.mark.parametrize("n,rows,m", [(1000, 100, 1500), (200000, 50000, 300000), (200000, 90000, 200000),
                                      (1 << 20, 3000, 200000)])
def test_one_way_edges(sg, n, rows, m):
    """Edges stored in one direction, to vertices most of which have no row: the
    same labels at every call, and those of the byte-width snapshot."""
    rng = np.random.default_rng(m)
    e = np.stack([rng.permutation(n)[:rows][rng.integers(0, rows, m)], rng.integers(0, n, m)], 1)
    g = sg.SparseMatrixV(n)
    g.insert_batch(e.astype(np.uint32))
    c = sg.CompactGraph(g)
    want = np.asarray(c.cc())
    for _ in range(3):
        assert np.array_equal(np.asarray(sg.CC(g)), want)
    c.close()
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("n,rows,m", [(300007, 300007, 196000), (1 << 20, 400000, 600000),
                                      (1 << 20, 200000, 220000)])
def test_one_way_edges_over_the_rounds(sg, n, rows, m, seed):
    """Enough rows for the sampled rounds, yet fewer than half of the vertices:
    what one round has joined the later ones keep, also behind vertices without a
    row."""
    rng = np.random.default_rng([m, seed])
    e = np.stack([rng.permutation(n)[:rows][rng.integers(0, rows, m)], rng.integers(0, n, m)], 1)
    g = sg.SparseMatrixV(n)
    g.insert_batch(e.astype(np.uint32))
    c = sg.CompactGraph(g)
    assert np.array_equal(np.asarray(sg.CC(g)), np.asarray(c.cc()))
    c.close()
    g.close()
