"""The row walks (pull gather, push, target marking) at the sizes where rows
change hands: lengths around the 128-bit id loads, the lanes per row, the
degree classes and the hub chunks, with the edge array ending at every
position of a load; and the compute kernel's bitmaps at their edges."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# around quads (4), 8 and 16 lanes of quads (32, 64), the classes (16, 64), hub chunks (256 on a small graph)
LENGTHS = (0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 35, 36, 63, 64, 65, 67, 68, 127, 128, 129, 255, 256, 257,
           511, 512, 513, 1500, 4096, 4097)
PR_TOL = 1e-12  # the oracle folds a row in order, the warp classes in a tree


def _graph(tail):
    """Rows of LENGTHS in a shuffled order, then `tail` edges in the last row (the edge count modulo 4 varies)."""
    rng = np.random.default_rng(7 + tail)
    V = 5000
    deg = np.zeros(V, dtype=np.int64)
    deg[rng.permutation(V - 1)[:len(LENGTHS)]] = LENGTHS
    deg[V - 1] = tail
    idx = np.concatenate(([0], np.cumsum(deg)[:-1])).astype(np.uint64)
    adj = np.concatenate([rng.choice(V, int(d), replace=False) for d in deg]).astype(np.uint32)
    return O.CSR(V, int(deg.sum()), idx, adj, None)


@pytest.mark.parametrize("tail", [0, 1, 2, 3])
@pytest.mark.parametrize("rounds", [1, 2, 3, 10])
@pytest.mark.parametrize("directed", [False, True])
def test_f32_rows_of_every_length(directed, rounds, tail):
    """PageRank's precision split over the same rows; supersteps 1 and 2 write the vertices without in-edges.
    Tolerances: a few FP32 roundings a superstep against FP64 (as the split's other tests), and the FP64 diagnostics
    against sums of the returned values."""
    import ipregel_b200 as ip
    g = _graph(tail)
    want, _, _ = O.run(g, "pagerank", "single_broadcast", rounds=rounds, directed=directed)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj, directed=directed)
    pr = ip.PageRankF32(graph)
    try:
        x, diag = pr.run(rounds=rounds)
        prev, _ = pr.run(rounds=rounds - 1)
    finally:
        pr.free()
        graph.free()
    assert np.max(np.abs(x - want) / want) <= 1e-5
    x, prev = x.astype(np.float64), prev.astype(np.float64)
    deg = np.diff(g.idx.astype(np.int64), append=g.E)
    np.testing.assert_allclose(diag[-1], [x.sum(), x[deg == 0].sum(), np.abs(x - prev).sum()], rtol=1e-12)


@pytest.mark.parametrize("tail", [0, 1, 2, 3])
@pytest.mark.parametrize("app,version,id_bits,variant", [
    ("pagerank", "single_broadcast", 32, ""), ("pagerank", "single_broadcast", 32, "staged"),
    ("cc", "single_broadcast", 32, ""), ("cc", "single_broadcast", 64, "")])
def test_rows_of_every_length(app, version, id_bits, variant, tail):
    import ipregel_b200 as ip
    g = _graph(tail)
    want, counts, _ = O.run(g, app, version, id_bytes=id_bits // 8)
    adj = g.adj if id_bits == 32 else g.adj.astype(np.uint64)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, adj, id_bytes=id_bits // 8)
    eng = ip.Engine(app, version, id_bits, variant=variant)
    eng.set_quiet(True)
    try:
        if app == "pagerank":
            eng.set_param("rounds", 10)
        # the default classes; classes of one lane a row up to a quad; every row above 3 edges a hub; small CTAs
        for tune in (dict(), dict(t0=4, t1=4096), dict(t0=2, t1=3), dict(block=64, t0=64, t1=200)):
            for order in (True, False):
                eng.set_order(order)
                eng.set_tuning(**tune)
                eng.attach(graph)
                res = eng.run()
                assert res.counts == [int(c) for c in counts], (tune, order)
                if app == "pagerank":
                    assert float(np.max(np.abs(res.values - want))) <= PR_TOL, (tune, order)
                else:
                    np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_tuning()
        eng.set_order(True)
        eng.release()
        graph.free()


@pytest.mark.parametrize("tail", [0, 1, 2, 3])
@pytest.mark.parametrize("app,version,id_bits,generic", [
    ("cc", "combiner", 32, False), ("cc", "spread", 32, False), ("cc", "single_broadcast_spread", 32, False),
    ("cc", "spread", 64, False), ("cc", "single_broadcast_spread", 64, False), ("cc", "spread", 32, True),
    ("sssp_weighted", "combiner", 32, False), ("sssp_weighted", "spread", 32, False), ("pagerank", "combiner", 32, False),
    ("pagerank", "spread", 32, True)])
def test_pushed_rows_of_every_length(app, version, id_bits, generic, tail):
    import ipregel_b200 as ip
    g = _graph(tail)
    rng = np.random.default_rng(tail)
    wgt = rng.integers(1, 256, g.E).astype(np.uint32) if app == "sssp_weighted" else None
    g = O.CSR(g.V, g.E, g.idx, g.adj, wgt)
    want, counts, _ = O.run(g, app, version, id_bytes=id_bits // 8)
    adj = g.adj if id_bits == 32 else g.adj.astype(np.uint64)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, adj, wgt=wgt, id_bytes=id_bits // 8)
    eng = ip.Engine(app, version, id_bits, generic)
    eng.set_quiet(True)
    try:
        if app == "pagerank":
            eng.set_param("rounds", 10)
        if app == "sssp_weighted":
            eng.set_param("source", 0)
        for tune in (dict(), dict(t0=4, t1=4096), dict(t0=2, t1=3), dict(block=64, t0=64, t1=200)):
            for order in (True, False):
                eng.set_order(order)
                eng.set_tuning(**tune)
                eng.attach(graph)
                res = eng.run()
                assert res.counts == [int(c) for c in counts], (tune, order)
                if app == "pagerank":
                    assert float(np.max(np.abs(res.values - want))) <= PR_TOL, (tune, order)
                else:
                    np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_tuning()
        eng.set_order(True)
        eng.release()
        graph.free()


@pytest.mark.parametrize("V", [1, 31, 32, 33, 127, 128, 129, 4095, 4097, 40_001, 700_001])
@pytest.mark.parametrize("app,version", [("cc", "combiner"), ("cc", "spread"), ("cc", "single_broadcast_spread"),
                                         ("sssp", "spread"), ("cc", "single_broadcast")])
def test_bitmap_edges(app, version, V):
    """Vertex counts around the words of the bitmaps, the steps of a warp and the batches of supersteps: a ring (the
    frontier of two vertices crosses every word) for the small ones, a random graph for the others."""
    import ipregel_b200 as ip
    if V <= 129:
        g = O.from_edges(V, [(i, (i + 1) % V) for i in range(V) if V > 1] + [((i + 1) % V, i) for i in range(V) if V > 2])
    else:
        g = O.gen_er(V, 3 * V, seed=V, undirected=True)
    want, counts, _ = O.run(g, app, version)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine(app, version)
    eng.set_quiet(True)
    try:
        if app == "sssp":
            eng.set_param("source", 0)
        for loop in (False, True):
            eng.set_graph_loop(loop)
            eng.attach(graph)
            for _ in range(2):
                res = eng.run()
                assert res.counts == [int(c) for c in counts]
                np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_graph_loop(False)
        eng.release()
        graph.free()


def test_users_of_one_graph_keep_their_classes(monkeypatch):
    """An engine and precision-split plans with other thresholds hold classes and hub tables of the same graph at
    the same time; running one after another has been made leaves its results bitwise as they were."""
    import ipregel_b200 as ip
    g = _graph(1)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("pagerank", "single_broadcast")
    eng.set_quiet(True)
    plans = []
    try:
        eng.set_param("rounds", 10)
        eng.attach(graph)
        first = eng.run().values.copy()
        runs = []
        for t0, t1 in ((16, 4096), (4, 100), (8, 40)):
            monkeypatch.setenv("IPG_PR_T0", str(t0))
            monkeypatch.setenv("IPG_PR_T1", str(t1))
            plans.append(ip.PageRankF32(graph))
            runs.append(plans[-1].run(rounds=10)[0].copy())
        np.testing.assert_array_equal(eng.run().values, first)
        for plan, x in zip(plans, runs):
            np.testing.assert_array_equal(plan.run(rounds=10)[0], x)
    finally:
        for plan in plans:
            plan.free()
        eng.release()
        graph.free()


@pytest.mark.parametrize("tail", [0, 1, 2, 3])
@pytest.mark.parametrize("app,version,id_bits,generic,symmetric", [
    ("cc", "combiner", 32, False, False), ("cc", "spread", 32, False, True), ("cc", "spread", 64, False, False),
    ("cc", "spread", 32, True, False), ("sssp_weighted", "combiner", 32, False, True),
    ("sssp_weighted", "spread", 32, False, False), ("pagerank", "combiner", 32, False, False)])
def test_pulled_rows_of_every_length(app, version, id_bits, generic, symmetric, tail):
    """Every superstep with an edge to deliver pulls (over the transpose, or over the rows of a symmetric graph)."""
    import ipregel_b200 as ip
    g = _graph(tail)
    rng = np.random.default_rng(tail)
    # the in-lists get the lengths: edges reversed, and both ways on the symmetric graph
    src, dst = g.adj.astype(np.int64), np.repeat(np.arange(g.V), np.diff(g.idx.astype(np.int64), append=g.E))
    if symmetric:
        src, dst = np.concatenate((src, dst)), np.concatenate((dst, src))
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    deg = np.bincount(src, minlength=g.V)
    idx = np.concatenate(([0], np.cumsum(deg)[:-1])).astype(np.uint64)
    wgt = (1 + (src * 31 + dst * 31 + src * dst) % 255).astype(np.uint32) if app == "sssp_weighted" else None
    g = O.CSR(g.V, len(src), idx, dst.astype(np.uint32), wgt)
    want, counts, _ = O.run(g, app, version, id_bytes=id_bits // 8)
    adj = g.adj if id_bits == 32 else g.adj.astype(np.uint64)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, adj, wgt=wgt, id_bytes=id_bits // 8, directed=not symmetric)
    if symmetric:
        graph.set_symmetric(True)
    eng = ip.Engine(app, version, id_bits, generic)
    eng.set_quiet(True)
    try:
        if app == "pagerank":
            eng.set_param("rounds", 10)
        if app == "sssp_weighted":
            eng.set_param("source", 0)
        for tune in (dict(), dict(t0=4, t1=4096), dict(t0=2, t1=3), dict(block=64, t0=64, t1=200)):
            for order in (True, False):
                eng.set_order(order)
                eng.set_tuning(pull_div=10 ** 9, **tune)
                eng.attach(graph)
                res = eng.run()
                assert res.counts == [int(c) for c in counts], (tune, order)
                if app == "pagerank":
                    assert float(np.max(np.abs(res.values - want))) <= PR_TOL, (tune, order)
                else:
                    np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_tuning()
        eng.set_order(True)
        eng.release()
        graph.free()
