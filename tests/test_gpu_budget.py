"""Work that fits a memory budget: what an update may take beside the graph
does not grow with the rows of the matrix or with the form that it takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    import __graft_entry__ as ge
    ge.build()
    import sstgraph_gb300
    return sstgraph_gb300


def device(e):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(e).astype(np.int32)).cuda()
    torch.cuda.synchronize()
    return t


# fewer pairs than rows: on the load's own path as many as its scratch allows
@pytest.mark.parametrize("n,b", [(1 << 22, 3000), (1 << 20, 40000), (1 << 20, 50000), (5000, 3000)])
def test_load_of_few_pairs(sg, n, b):
    e = np.random.default_rng(b).integers(0, n, (b, 2))
    e = e[e[:, 0] != e[:, 1]]
    g = sg.SparseMatrixV(n)
    empty = g.get_memory_size()
    g.close()
    # the general sequence's planning, rounded up and over, and its staging
    g = sg.SparseMatrixV(n, hbm_budget_bytes=empty + 550 * b + (3 << 20))
    g.insert_batch(device(e))
    k = np.unique(e[:, 0] * n + e[:, 1])
    assert g.M() == len(k)
    off, cols = g.csr()
    assert np.array_equal(np.repeat(np.arange(n), np.diff(off.astype(np.int64))) * n + cols, k)
    g.close()


# The least beside the graph that each was found to fit when one sequence of
# launches took every batch and sort tiles held 4096 keys.
@pytest.mark.parametrize("b,least", [(1, 1236928), (100, 1256384), (700, 1516224),
                                     (20000, 9527808), (262145, 131383296),
                                     (600000, 261840896), (1 << 20, 423149568)])
@pytest.mark.parametrize("plan", [True, False])
def test_batches_of_any_form(sg, b, least, plan):
    n = 1 << 20
    first = device([[5, 7], [7, 5]])
    e = device(np.random.default_rng(2).integers(0, n, (b, 2)))
    g = sg.SparseMatrixV(n)
    empty = g.get_memory_size()
    g.close()
    g = sg.SparseMatrixV(n, hbm_budget_bytes=empty + least)
    g.set_plan_graphs(plan)
    g.insert_batch(first)  # no graph without segments: that is a load
    g.release_scratch()
    g.insert_batch(e)
    assert g.M() > b // 2
    g.close()


# What each traversal keeps on an RMAT graph of 2^18 vertices and 2^21 drawn
# edges, when its levels were launches of their own.
@pytest.mark.parametrize("name,most", [("bfs", 22572280), ("pr", 23662752), ("cc", 15095800),
                                       ("bc", 29828512), ("tc", 41834720)])
def test_traversal_buffers(sg, name, most):
    import torch
    run = {"bfs": lambda: sg.BFS(g, 1), "pr": lambda: sg.PR_S(g, 2), "cc": lambda: sg.CC(g),
           "bc": lambda: sg.BC(g, 1), "tc": lambda: sg.TC(g)}[name]
    e = torch.empty((8 << 18, 2), dtype=torch.int32, device="cuda")
    sg.gen_rmat(18, 8 << 18, out=e)
    torch.cuda.synchronize()
    e = torch.cat([e, e.flip(1)]).contiguous()
    torch.cuda.synchronize()
    g = sg.SparseMatrixV(1 << 18)
    g.insert_batch(e)
    g.release_scratch()
    before = g.get_memory_size()
    run()
    assert g.get_memory_size() - before <= most
    g.close()
