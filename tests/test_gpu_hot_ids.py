"""The flagged copy of the in-lists (IPG_SB_HOT_KB) is read in whole groups of four ids like the lists themselves."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [0, 1, 2, 3])
def test_flagged_copy_holds_whole_groups(tail, monkeypatch):
    import ipregel_b200 as ip
    rng = np.random.default_rng(tail)
    V = 300
    deg = rng.integers(0, 40, V)
    deg[-1] = 0
    deg[-1] = 4 + (tail - int(deg.sum())) % 4  # the edge count modulo 4 is tail
    idx = np.concatenate(([0], np.cumsum(deg)[:-1])).astype(np.uint64)
    adj = np.concatenate([rng.choice(V, int(d), replace=False) for d in deg]).astype(np.uint32)
    g = O.CSR(V, int(deg.sum()), idx, adj, None)
    assert g.E % 4 == tail
    want, counts, _ = O.run(g, "cc", "single_broadcast")
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("cc", "single_broadcast")
    eng.set_quiet(True)
    used = {}
    try:
        eng.set_order(False)
        for kb in ("65536", "0", "65536"):  # the first attach also builds the graph's classes
            monkeypatch.setenv("IPG_SB_HOT_KB", kb)
            eng.release()
            eng.attach(graph)
            used[kb] = ip.hbm_in_use()
            res = eng.run()
            assert res.counts == [int(c) for c in counts]
            np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
        assert used["65536"] - used["0"] == 4 * ((g.E + 3) // 4 * 4)
    finally:
        eng.set_order(True)
        eng.release()
        graph.free()
