"""Pairs loaded into a graph without segments (from 2049 pairs on a path of
its own), against the CPU oracle, the structural check and the general path."""
import numpy as np
import pytest

import oracle
from pma_check import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    import __graft_entry__ as ge
    ge.build()
    import sstgraph_gb300
    return sstgraph_gb300


def same(g, o, like=None):
    oo, co = o.csr()
    og, cg = g.csr()
    assert g.M() == o.M()
    assert np.array_equal(og, oo) and np.array_equal(cg, co)
    assert np.array_equal(g.degrees(), o.degrees())
    # a low fill leaves leaves empty, on the general path too: the same ones
    want = check(like) if like else []
    errs = check(g, None if want else (oo, co))
    assert errs == want, errs[:5]


def pairs(rng, n, b, shape):
    """b pairs with repeats, self-loops and ids out of range"""
    e = rng.integers(0, n, (b, 2)).astype(np.uint32)
    if shape == "hub":      # one row of most ids, rows of one leaf and just above
        e[: b // 2, 0] = n - 1
        for i, d in enumerate((31, 32, 33, 64, 65)):
            e[b // 2 + 100 * i: b // 2 + 100 * i + d, 0] = i
    elif shape == "equal":  # runs of equal keys across tiles
        e[:, 0] %= 7
        e[:, 1] %= 5
    elif shape == "none":   # no pair is kept
        e[:, 1] = e[:, 0]
    if shape != "none":
        e[::11, 1] = e[::11, 0]
        e[::17] = e[0]
        e[5::1001, 0] = n + 3
    return e


@pytest.mark.parametrize("b", [2048, 2049, 4097, 16384, 18433, 40001, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("shape", ["even", "hub", "equal", "none"])
def test_load(sg, b, shape):
    rng = np.random.default_rng(b)
    n = 4999
    e = pairs(rng, n, b, shape)
    o = oracle.OracleGraph(n)
    o.insert_batch(e[e.max(1) < n])
    for fill in (0.7, 0.02):
        g = sg.SparseMatrixV(n, grow_fill=fill, initial_slots=64 if fill < 0.1 else 0)
        assert g.insert_batch(e) == int((e.max(1) >= n).sum())
        w = None
        if fill < 0.1:
            w = sg.SparseMatrixV(n, grow_fill=fill, weighted=True)  # the general path
            w.insert_batch(e)
        same(g, o, w)
        # the loaded graph takes updates
        u = rng.integers(0, n, (5000, 2)).astype(np.uint32)
        g.insert_batch(u)
        g.remove_batch(e[: b // 3][e[: b // 3].max(1) < n])
        o2 = oracle.OracleGraph(n)
        o2.insert_batch(e[e.max(1) < n])
        o2.insert_batch(u)
        o2.remove_batch(e[: b // 3][e[: b // 3].max(1) < n])
        if w:
            oo, co = o2.csr()
            og, cg = g.csr()
            assert np.array_equal(og, oo) and np.array_equal(cg, co)
            w.close()
        else:
            same(g, o2)
        g.close()


@pytest.mark.parametrize("loops", [False, True])
def test_load_as_the_general_path_does(sg, loops):
    """Same sizes, edges and leaf fill as the general path, which weighted
    graphs take; a rectangular matrix; pairs at 4-byte alignment."""
    import torch
    rng = np.random.default_rng(3)
    n, width, b = 3001, 70000, 100000
    e = np.stack([rng.integers(0, n, b) ** 2 // n, rng.integers(0, width, b)], 1).astype(np.uint32)
    buf = torch.zeros(2 * b + 1, dtype=torch.int32, device="cuda")
    buf[1:] = torch.from_numpy(e.astype(np.int32).reshape(-1)).cuda()
    g = sg.SparseMatrixV(n, width, keep_self_loops=loops)
    w = sg.SparseMatrixV(n, width, keep_self_loops=loops, weighted=True)
    g.insert_batch(buf[1:].view(b, 2))
    w.insert_batch(e)
    assert g.M() == w.M()
    for x, y in zip(g.csr(), w.csr()):
        assert np.array_equal(x, y)
    assert np.array_equal(g.degrees(), w.degrees())
    g.close()
    w.close()


# the records in one allocation, in two, and in one again
@pytest.mark.parametrize("n", [1, 63000, 66000, 120000, 132000])
def test_records_of_any_size(sg, n):
    e = np.array([[0, n - 1], [n // 2, 0], [n - 1, n - 1], [n - 1, n // 3]], np.uint32)
    e = e[e[:, 0] != e[:, 1]]
    for _ in range(3):
        g = sg.SparseMatrixV(n)
        o = oracle.OracleGraph(n)
        if len(e):
            assert g.insert_batch(e) == 0
            o.insert_batch(e)
        h = g.copy()
        g.close()
        same(h, o)
        h.close()
