"""Graphs over a caller's device arrays (ipg_graph_from_device): ids and weights that end inside a group of four, or do not
begin on a 16-byte boundary, are walked without 128-bit loads.  Every walk over them, on the graph's own numbering."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# around the lanes and unrolled steps of the walks (8, 16, 32 lanes x 4), the classes (16, 64) and hub chunks (256)
LENGTHS = (0, 1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 512, 513, 1500, 4097)
PR_TOL = 1e-12  # the oracle folds a row in order, the walks in trees


def _graph(tail, both=False):
    """Rows of LENGTHS and more in a shuffled order, with weights; `tail` of the last row makes E modulo 4 vary.
    both: every edge in both directions."""
    rng = np.random.default_rng(11 + tail)
    V = 5000
    deg = np.zeros(V, dtype=np.int64)
    deg[rng.permutation(V - 1)[:len(LENGTHS)]] = LENGTHS
    deg[V - 1] = tail
    src = np.repeat(np.arange(V), deg)
    dst = np.concatenate([rng.choice(V, int(d), replace=False) for d in deg])
    if both:
        src, dst = np.concatenate((src, dst)), np.concatenate((dst, src))
        key = np.unique(src * V + dst)
        src, dst = key // V, key % V
        deg = np.bincount(src, minlength=V)
    wgt = (1 + (src * 31 + dst * 31 + src * dst) % 255).astype(np.uint32)
    idx = np.concatenate(([0], np.cumsum(deg)[:-1])).astype(np.uint64)
    return O.CSR(V, len(src), idx, dst.astype(np.uint32), wgt)


class _Caller:
    """A graph over arrays of exactly its size whose ids and weights begin `off` words into an allocation."""

    def __init__(self, g, off, weighted, symmetric):
        import ipregel_b200 as ip

        def up(a, o):
            d = ip.DeviceArray(a.size + o, a.dtype)
            d.from_host(np.concatenate((np.zeros(o, a.dtype), a)))
            return d

        row = up(np.append(g.idx, np.uint64(g.E)).astype(np.uint64), 0)
        adj, wgt = up(g.adj, off), up(g.wgt, off) if weighted else None
        self.keep = (row, adj, wgt)
        h = ctypes.c_void_p()
        rc = ip.runtime().ipg_graph_from_device(g.V, g.E, row.ptr, adj.ptr + 4 * off, 4, wgt.ptr + 4 * off if wgt else None,
                                                4 if wgt else 0, 0, 0, ctypes.byref(h))
        assert rc == 0, ip.runtime().ipg_last_error()
        self.graph = ip.Graph(h.value)
        if symmetric:
            self.graph.set_symmetric(True)
        q = ctypes.c_int()
        assert ip.runtime().ipg_graph_quads(ctypes.c_void_p(h.value), 0, ctypes.byref(q)) == 0
        assert q.value == (off == 0 and g.E % 4 == 0)

    def free(self):
        self.graph.free()
        for d in self.keep:
            if d is not None:
                d.free()


@pytest.mark.parametrize("tail,off", [(0, 0), (1, 0), (2, 0), (3, 0), (0, 1), (1, 3)])
@pytest.mark.parametrize("app,version,pull", [
    ("cc", "combiner", False), ("cc", "spread", False), ("cc", "spread", True), ("cc", "single_broadcast", False),
    ("cc", "single_broadcast_spread", False), ("sssp_weighted", "spread", False), ("sssp_weighted", "combiner", True),
    ("pagerank", "single_broadcast", False), ("pagerank", "combiner", True)])
def test_rows_of_a_caller(app, version, pull, tail, off):
    import ipregel_b200 as ip
    g = _graph(tail, both=pull)
    want, counts, _ = O.run(g, app, version)
    c = _Caller(g, off, app == "sssp_weighted", pull)
    eng = ip.Engine(app, version)
    eng.set_quiet(True)
    try:
        if app == "pagerank":
            eng.set_param("rounds", 10)
        if app == "sssp_weighted":
            eng.set_param("source", 0)
        eng.set_order(False)
        for tune in (dict(), dict(t0=2, t1=3), dict(block=64, t0=64, t1=200)):
            eng.set_tuning(pull_div=10 ** 9 if pull else 0, **tune)
            eng.attach(c.graph)
            res = eng.run()
            assert res.counts == [int(x) for x in counts], tune
            if app == "pagerank":
                assert float(np.max(np.abs(res.values - want))) <= PR_TOL, tune
            else:
                np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_tuning()
        eng.set_order(True)
        eng.release()
        c.free()


@pytest.mark.parametrize("tail,off", [(0, 0), (1, 0), (2, 0), (3, 0), (0, 1), (1, 3)])
def test_f32_rows_of_a_caller(tail, off, monkeypatch):
    """A few FP32 roundings a superstep against FP64, as the split's other tests."""
    import ipregel_b200 as ip
    monkeypatch.setenv("IPG_ORDER", "0")
    g = _graph(tail)
    want, _, _ = O.run(g, "pagerank", "single_broadcast", rounds=10)
    c = _Caller(g, off, False, False)
    plan = ip.PageRankF32(c.graph)
    try:
        for compensated in (True, False):
            x, _ = plan.run(rounds=10, compensated=compensated)
            assert np.max(np.abs(x - want) / want) <= (1e-5 if compensated else 1e-4)
    finally:
        plan.free()
        c.free()


def test_marking_with_two_ctas_per_sm():
    """Spread + single_broadcast on more than 2^23 edges, where the marking kernel is the one with two CTAs per SM."""
    import ipregel_b200 as ip
    g = O.gen_rmat(19, 10, seed=4, undirected=True)
    assert g.E > 1 << 23
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("cc", "single_broadcast_spread")
    eng.set_quiet(True)
    want, counts, _ = O.run(g, "cc", "single_broadcast_spread")
    try:
        for order in (True, False):
            eng.set_order(order)
            eng.attach(graph)
            res = eng.run()
            assert res.counts == [int(x) for x in counts]
            np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_order(True)
        eng.release()
        graph.free()
