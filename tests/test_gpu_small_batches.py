"""Batches up to 1024 pairs (their own three launches) and just above, against
the CPU oracle and the structural check, and against the same pairs given in
batches of the general path."""
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


def same(g, o):
    oo, co = o.csr()
    og, cg = g.csr()
    assert g.M() == o.M()
    assert np.array_equal(og, oo) and np.array_equal(cg, co)
    assert np.array_equal(g.degrees(), o.degrees())
    errs = check(g, (oo, co))
    assert not errs, errs[:5]


def batch(rng, o, n, b, shape):
    """b pairs with repeats, self-loops, present edges and ids out of range"""
    e = rng.integers(0, n, (b, 2)).astype(np.uint32)
    if shape == "hub":            # one long row: windows, resizes, shared leaves
        e[: b // 2, 0] = 3
    elif shape == "run":          # neighbouring ids of a few rows: one leaf's worth
        e[:, 0] %= 4
        e[:, 1] = (rng.integers(0, n - b) + np.arange(b)) % n
    e[b // 2:][:: 7] = e[: b - b // 2][:: 7]
    e[::11, 1] = e[::11, 0]
    if b > 5:
        e[5] = (n, 1)
        e[4] = (1, 0xFFFFFFFF)
    return e


def valid(e, n):
    return e[(e[:, 0] < n) & (e[:, 1] < n)]


# the sort's runs of 32 and its powers of two, two items a thread, the limit
@pytest.mark.parametrize("b", [1, 2, 31, 32, 33, 64, 65, 127, 257, 511, 512, 513, 1023, 1024, 1025])
@pytest.mark.parametrize("shape", ["any", "hub", "run"])
def test_stream(sg, b, shape):
    n = 3000
    rng = np.random.default_rng(b)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    for step in range(8):
        e = batch(rng, o, n, b, shape)
        bad = len(e) - len(valid(e, n))
        assert g.insert_batch(e) == bad
        o.insert_batch(valid(e, n))
        if step % 2:
            r = np.concatenate([batch(rng, o, n, max(b // 3, 1), shape), e[: b // 2 + 1]])[:b]
            assert g.remove_batch(r) == len(r) - len(valid(r, n))
            o.remove_batch(valid(r, n))
        same(g, o)


def test_empties_and_refills_rows(sg):
    """rows of one leaf and of many, emptied and filled again in small steps"""
    n = 2000
    rng = np.random.default_rng(4)
    base = np.concatenate([np.stack([np.full(k, v), rng.choice(n, k, replace=False)], 1)
                           for v, k in ((1, 1500), (2, 400), (3, 65), (4, 33), (5, 32), (6, 3))])
    base = base[base[:, 0] != base[:, 1]].astype(np.uint32)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    for op in ("insert", "remove", "insert"):
        order = rng.permutation(len(base))
        for i in range(0, len(base), 300):
            part = base[order[i:i + 300]]
            getattr(g, op + "_batch")(part)
            getattr(o, op + "_batch")(part)
            same(g, o)


def test_slab_runs_full(sg):
    """repacks in the middle of small batches: the merges run before it, the
    resizes after it"""
    n = 4000
    rng = np.random.default_rng(8)
    g = sg.SparseMatrixV(n, initial_slots=4096)
    o = oracle.OracleGraph(n)
    for _ in range(60):
        e = rng.integers(0, n, (1000, 2)).astype(np.uint32)
        e[:300, 0] %= 5
        g.insert_batch(e)
        o.insert_batch(e)
    same(g, o)


def test_equals_the_general_path(sg):
    """the same stream in batches of 1024 and of 1025 to 3000"""
    n = 3000
    rng = np.random.default_rng(12)
    a, c = sg.SparseMatrixV(n), sg.SparseMatrixV(n)
    for op in ("insert", "insert", "remove", "insert"):
        e = rng.integers(0, n, (6000, 2)).astype(np.uint32)
        e[::3, 0] %= 3
        for i in range(0, len(e), 1024):
            getattr(a, op + "_batch")(e[i:i + 1024])
        for i in range(0, len(e), 3000):
            getattr(c, op + "_batch")(e[i:i + 3000])
        for x, y in zip(a.csr(), c.csr()):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("offset", [0, 1])
def test_device_and_pinned_pairs(sg, offset):
    """device, pinned and pageable pairs, on and off the 8-byte boundary"""
    torch = pytest.importorskip("torch")
    n, b = 3000, 700
    rng = np.random.default_rng(3)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)
    for kind in ("cuda", "pinned", "host"):
        e = rng.integers(0, n, (b, 2)).astype(np.uint32)
        buf = torch.zeros(2 * b + 1, dtype=torch.int32)
        if kind == "pinned":
            buf = buf.pin_memory()
        if kind == "cuda":
            buf = buf.cuda()
        buf[offset:offset + 2 * b].copy_(torch.from_numpy(e.view(np.int32).reshape(-1)))
        if kind == "cuda":
            torch.cuda.synchronize()
        g.insert_batch(buf[offset:offset + 2 * b])
        o.insert_batch(e)
        same(g, o)


# rows whose tasks the cluster applies, and whose tasks take grids (1024 leaves
# read and written in all), grown past a resize and shrunk below one
@pytest.mark.parametrize("cap", [1 << 13, 1 << 14, 1 << 15, 1 << 17])
def test_long_row(sg, cap):
    n, b = 2 * cap, 900
    rng = np.random.default_rng(cap)
    p = rng.permutation(n).astype(np.uint32)
    g, o = sg.SparseMatrixV(n), oracle.OracleGraph(n)

    def step(op, cols):
        e = np.stack([np.full(len(cols), 3, np.uint32), cols], 1)
        other = rng.integers(0, n, (1000 - b, 2)).astype(np.uint32) if len(cols) <= b else e[:0]
        e = np.concatenate([e, other])
        e = e[e[:, 0] != e[:, 1]]
        for m in (g, o):
            getattr(m, op)(e)

    at = int(0.84 * cap)
    step("insert_batch", p[:at])
    for _ in range(cap // 4 // b + 3 if cap <= 1 << 15 else 4):
        step("insert_batch", p[at:at + b])
        at += b
    same(g, o)
    keep = int(0.2 * 2 * cap) + 2 * b
    step("remove_batch", p[keep:at])
    for _ in range(4):
        step("remove_batch", p[keep - b:keep])
        keep -= b
    same(g, o)
    g.close()
