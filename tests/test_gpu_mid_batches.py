"""Batches of up to 4096 pairs past the small form (their planning steps in one
block each) and just above, replayed, launched directly and as a sequence of
batches, against the CPU oracle and the structural check."""
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


def batch(rng, n, b, shape):
    e = rng.integers(0, n, (b, 2)).astype(np.uint32)
    if shape == "hub":        # one long row: windows, resizes, shared leaves
        e[: b // 2, 0] = 3
    elif shape == "run":      # whole leaves of a few rows
        e[:, 0] %= 3
        e[:, 1] = (rng.integers(0, n) + np.arange(b) // 2) % n
    e[::11, 1] = e[::11, 0]
    e[1::13] = e[0]
    return e


@pytest.mark.parametrize("b", [1025, 1792, 3001, 4096, 4097])
@pytest.mark.parametrize("shape", ["even", "hub", "run"])
@pytest.mark.parametrize("mode", [True, False])
def test_mid_batches(sg, b, shape, mode):
    n = 3000
    rng = np.random.default_rng(b)
    g = sg.SparseMatrixV(n, initial_slots=64)
    g.set_plan_graphs(mode)
    o = oracle.OracleGraph(n)
    seed = rng.integers(0, n, (1000, 2)).astype(np.uint32)
    g.insert_batch(seed)
    o.insert_batch(seed)
    for i in range(6):
        e = batch(rng, n, b, shape)
        if i % 3 == 2:
            e = np.concatenate([e[: b // 2], o.sample_edges(b - b // 2, seed=i)])
            assert g.remove_batch(e) == 0
            o.remove_batch(e)
        else:
            assert g.insert_batch(e) == 0
            o.insert_batch(e)
        same(g, o)
    r = o.sample_edges(b, seed=9)
    k = batch(rng, n, b // 2, shape)
    g.update_batches([r, k], [0, 1])
    o.remove_batch(r)
    o.insert_batch(k)
    same(g, o)
    g.close()
