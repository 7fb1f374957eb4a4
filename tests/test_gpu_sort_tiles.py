"""The key sort at the edges of its one-block forms, of its tiles (1024, 2048 and
4096 keys) and
of the groups of 8, 64 and 512 tiles whose digit counts a pass adds up, through
the bulk insert (keys) and the batched form (keys with operations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    import __graft_entry__ as ge
    ge.build()
    import sstgraph_gb300
    return sstgraph_gb300


def pairs(n, b, seed):
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, (b, 2)).astype(np.uint32)
    e[: b // 3, 0] = 7           # one digit for a third of the keys
    return e


def edges(n, *es):
    k = np.concatenate([e[:, 0].astype(np.uint64) * n + e[:, 1] for e in es])
    k = np.unique(k)
    return k[k // n != k % n]


def of(g):
    off, cols = g.csr()
    rows = np.repeat(np.arange(g.rows, dtype=np.uint64), np.diff(off.astype(np.int64)))
    return rows * g.rows + cols


@pytest.mark.parametrize("b", [1025, 2048, 2049, 4095, 4096, 4097, 7 * 1024 + 1, 8 * 1024, 8 * 1024 + 1, 64 * 1024, 64 * 1024 + 1,
                               1 << 18, (1 << 18) + 1, 448 * 2048, 448 * 2048 + 1,
                               512 * 4096, 512 * 4096 + 1, 1100 * 4096 + 77])
@pytest.mark.parametrize("n", [60000, 1 << 20])
def test_keys(sg, b, n):
    e, f = pairs(n, b, b), pairs(n, b // 2, b + 1)
    g = sg.SparseMatrixV(n)
    g.insert_batch(e)                    # a load
    assert np.array_equal(of(g), edges(n, e))
    g.insert_batch(f)                    # an update
    assert np.array_equal(of(g), edges(n, e, f))
    g.close()


@pytest.mark.parametrize("b", [1025, 8 * 2048, 8 * 2048 + 1, 64 * 2048 + 1, 448 * 2048,
                               448 * 2048 + 1, 512 * 4096 + 1])
def test_keys_with_values(sg, b):
    n = 50000
    e = pairs(n, b, b)
    a, r, c = e[: b // 2], e[b // 4: b // 4 * 3], e[b // 2:]
    g = sg.SparseMatrixV(n)
    g.update_batches([a, r, c], [1, 0, 1])   # b + b / 2 pairs, the last operation wins
    want = np.setdiff1d(edges(n, a), edges(n, r))
    assert np.array_equal(of(g), np.union1d(want, edges(n, c)))
    g.close()


@pytest.mark.parametrize("one_by_one", [False, True])
@pytest.mark.parametrize("n", [1 << 10, 1000])
@pytest.mark.parametrize("loops", [False, True])
def test_dropped_pairs(sg, loops, n, one_by_one):
    """Self-loops (of row 0 too), ids out of range and edges given many times,
    on rows and columns that fill their bits and that do not."""
    b = 20000
    rng = np.random.default_rng(1)
    es = [rng.integers(0, n, (b, 2)).astype(np.uint32) for _ in range(5)]
    for e in es:
        e[::9] = 0
        e[1::9, 1] = e[1::9, 0]
        e[2::9, 0] = n
        e[3::9] = (0, 1)
    ops = [1, 0, 1, 0, 1]
    g = sg.SparseMatrixV(n, keep_self_loops=loops)
    bad = sum(int((e.max(1) >= n).sum()) for e in es)
    if one_by_one:
        assert sum((g.insert_batch if op else g.remove_batch)(e)
                   for e, op in zip(es, ops)) == bad
    else:
        assert g.update_batches(es, ops) == bad
    have = np.zeros(n * n, bool)
    for e, op in zip(es, ops):
        e = e[e.max(1) < n].astype(np.int64)
        have[e[:, 0] * n + e[:, 1]] = op
    if not loops:
        have[np.arange(n) * n + np.arange(n)] = False
    assert np.array_equal(of(g), np.flatnonzero(have).astype(np.uint64))
    g.close()


def test_batches_with_ids_of_64_bits(sg):
    """Rows and columns of 32 bits: no bit of a key is free for its operation."""
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 120 << 30:
        pytest.skip("the vertex records take 34 GB")
    n, w = (1 << 31) + 5, 0xfffffff0
    rng = np.random.default_rng(2)
    a = np.stack([rng.integers(0, n, 5000), rng.integers(0, w, 5000)], 1).astype(np.uint32)
    a[:3] = [(0, 0), (n - 1, w - 1), (n - 1, 0)]
    r = a[1::2].copy()
    g = sg.SparseMatrixV(n, w)
    assert g.update_batches([a, r, a[3::4]], [1, 0, 1]) == 0
    want = np.ones(5000, bool)
    want[1::2] = False
    want[3::4] = True
    want[0] = False  # a self-loop
    assert np.array_equal(np.asarray(g.has_batch(a)).astype(bool), want)
    assert g.M() == int(want.sum())
    g.close()
