"""A run that ends early: by the superstep bound, with supersteps enqueued beyond it that must do nothing."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _path(n):
    """Every vertex of a two-way path improves its label in every superstep until the ends have met, so the
    frontier (or the target set) stays near n."""
    return O.from_edges(n, [(i, i + 1) for i in range(n - 1)] + [(i + 1, i) for i in range(n - 1)])


@pytest.mark.parametrize("bound", [1, 3, 9])
@pytest.mark.parametrize("version", ["single_broadcast_spread", "spread", "combiner", "single_broadcast"])
@pytest.mark.parametrize("loop", [False, True])
def test_bounded_run_then_full(version, bound, loop, monkeypatch):
    import ipregel_b200 as ip
    g = _path(200)
    want, counts, _ = O.run(g, "cc", version)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("cc", version)
    eng.set_quiet(True)
    try:
        eng.set_graph_loop(loop)
        eng.attach(graph)
        monkeypatch.setenv("IPG_MAX_SUPERSTEPS", str(bound))
        with pytest.raises(ip.IPregelError, match="superstep limit"):
            eng.run()
        assert eng.counts() == [int(c) for c in counts[:bound]]
        monkeypatch.setenv("IPG_MAX_SUPERSTEPS", "20000")
        if loop:  # a captured loop holds the bound it was made with
            eng.attach(graph)
        res = eng.run()
        assert res.counts == [int(c) for c in counts]
        np.testing.assert_array_equal(res.values.astype(np.uint64), want.astype(np.uint64))
    finally:
        eng.set_graph_loop(False)
        eng.release()
        graph.free()


@pytest.mark.parametrize("version", ["combiner", "spread", "single_broadcast", "single_broadcast_spread"])
def test_bound_of_no_supersteps(version, monkeypatch):
    """The host-driven loop runs nothing under a bound of 0: no count, and the values as they were initialised."""
    import ipregel_b200 as ip
    g = _path(40)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("cc", version)
    eng.set_quiet(True)
    try:
        eng.attach(graph)
        before = eng.values().copy()
        monkeypatch.setenv("IPG_MAX_SUPERSTEPS", "0")
        with pytest.raises(ip.IPregelError, match="superstep limit"):
            eng.run()
        assert eng.counts() == []
        np.testing.assert_array_equal(eng.values(), before)
    finally:
        eng.release()
        graph.free()


def test_compact_unless():
    """The compaction between the engine's kernels: as ipg_compact while the flag is 0, and nothing appended, summed
    or cleared while it is not."""
    import ipregel_b200 as ip
    V = 1000
    deg = np.arange(V, dtype=np.uint64) % 40
    bits = np.random.default_rng(3).integers(0, 1 << 32, (V + 31) // 32, dtype=np.uint32)
    ids = np.flatnonzero(np.unpackbits(bits.view(np.uint8), bitorder="little")[:V])

    def up(a):
        d = ip.DeviceArray(a.size, a.dtype)
        d.from_host(a)
        return d

    row = up(np.concatenate(([0], np.cumsum(deg))).astype(np.uint64))
    for skip in (0, 1):
        flag, bm = up(np.array([skip], dtype=np.uint64)), up(bits)
        lists = [up(np.full(V, 7, dtype=np.uint32)) for _ in range(3)]
        cnt, edges = up(np.zeros(4, dtype=np.uint32)), up(np.zeros(3, dtype=np.uint64))
        f = ip.runtime().ipg_compact_unless
        f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64,
                      ctypes.c_uint64] + [ctypes.c_void_p] * 5 + [ctypes.c_int, ctypes.c_void_p]
        rc = f(flag.ptr, bm.ptr, V, row.ptr, 8, 24, *[x.ptr for x in lists], cnt.ptr, edges.ptr, 1, None)
        assert rc == 0
        for k, (lo, hi) in enumerate(((0, 8), (9, 24), (25, 1 << 30))):
            want = ids[(deg[ids] >= lo) & (deg[ids] <= hi)]
            if skip:
                assert cnt.to_host()[k] == 0 and edges.to_host()[k] == 0 and (lists[k].to_host() == 7).all()
            else:
                assert cnt.to_host()[k] == want.size and edges.to_host()[k] == deg[want].sum()
                np.testing.assert_array_equal(np.sort(lists[k].to_host()[:want.size]), want)
        np.testing.assert_array_equal(bm.to_host(), bits if skip else np.zeros_like(bits))


@pytest.mark.parametrize("version", ["combiner", "spread", "single_broadcast", "single_broadcast_spread"])
@pytest.mark.parametrize("n", [2, 40])
def test_total_time_is_the_supersteps(version, n, capfd):
    """The reported total is the sum of the supersteps' durations, without those enqueued beyond the end that do
    nothing (the durations are printed to a microsecond)."""
    import ipregel_b200 as ip
    g = _path(n)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    eng = ip.Engine("cc", version)
    try:
        eng.set_quiet(False)
        eng.attach(graph)
        res = eng.run()
        ctypes.CDLL(None).fflush(None)
        out = capfd.readouterr().out
        times = [float(x.split(":")[1]) for x in out.splitlines() if x.startswith("Superstep") and "Duration" in x]
        assert len(times) == len(res.counts) and min(times) >= 0
        assert abs(res.seconds - sum(times)) <= 0.6e-6 * len(times)
    finally:
        eng.set_quiet(True)
        eng.release()
        graph.free()
