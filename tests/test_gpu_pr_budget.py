"""The FP32 PageRank plan under a memory budget: without room for its list of short rows it runs all the same."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds", [0, 1, 2, 10])
@pytest.mark.parametrize("short_of", [1, 1 << 14])
def test_plan_without_its_list_of_short_rows(short_of, rounds):
    import ipregel_b200 as ip
    g = O.gen_rmat(14, 8, seed=6, undirected=False)  # many vertices without in-edges, some without out-edges
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj, directed=True, need_in=True)
    first = second = None
    try:
        first = ip.PageRankF32(graph)  # also makes the copy, its classes and hub table
        x, diag = first.run(rounds=rounds)
        used = ip.hbm_in_use()
        first.free()
        # the list is made last, and its scratch after it: first the one, then the other does not fit
        ip.set_hbm_budget(used - short_of)
        second = ip.PageRankF32(graph)
        ip.set_hbm_budget(0)
        assert ip.hbm_in_use() < used
        y, diag2 = second.run(rounds=rounds)
        np.testing.assert_array_equal(y, x)
        np.testing.assert_allclose(diag2, diag, rtol=1e-12, atol=1e-18)
    finally:
        ip.set_hbm_budget(0)
        for p in (first, second):
            if p is not None:
                p.free()
        graph.free()
