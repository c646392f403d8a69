"""A graph's degree classes and hub tables stay while somebody holds them: many users with thresholds of their own, and a
memory budget that has no room for another set."""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


class _Bins(ctypes.Structure):
    _fields_ = [("d_list", ctypes.c_void_p * 3), ("count", ctypes.c_uint64 * 3), ("edges", ctypes.c_uint64 * 3),
                ("t0", ctypes.c_uint64), ("t1", ctypes.c_uint64)]


class _Hubs(ctypes.Structure):
    _fields_ = [("d_hub", ctypes.c_void_p), ("hubs", ctypes.c_uint64), ("d_owner", ctypes.c_void_p),
                ("chunks", ctypes.c_uint64), ("edges", ctypes.c_uint64)]


def _lib():
    import ipregel_b200 as ip
    L = ip.runtime()
    vp, u64 = ctypes.c_void_p, ctypes.c_uint64
    L.ipg_graph_bins.argtypes = [vp, ctypes.c_int, u64, u64, vp]
    L.ipg_graph_hubs.argtypes = [vp, ctypes.c_int, u64, u64, vp]
    L.ipg_graph_hold.argtypes = [vp, vp, ctypes.POINTER(vp)]
    L.ipg_hold_release.argtypes = [vp]
    L.ipg_hold_release.restype = None
    return L


def _bins(graph, t0, t1):
    b = _Bins()
    return _lib().ipg_graph_bins(graph.handle, 0, t0, t1, ctypes.byref(b)), b


def _hubs(graph, hub_min, chunk):
    h = _Hubs()
    return _lib().ipg_graph_hubs(graph.handle, 0, hub_min, chunk, ctypes.byref(h)), h


def _hold(graph, d_set):
    p = ctypes.c_void_p()
    assert _lib().ipg_graph_hold(graph.handle, d_set, ctypes.byref(p)) == 0
    return p


def test_held_sets_stay():
    import ipregel_b200 as ip
    g = O.gen_rmat(12, 16, seed=3, undirected=True)
    deg = np.diff(g.idx.astype(np.int64), append=g.E)
    base = ip.hbm_in_use()
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    try:
        rc, b = _bins(graph, 8, 40)
        assert rc == 0
        rc, h = _hubs(graph, 100, 64)
        assert rc == 0
        holds = [_hold(graph, b.d_list[0]), _hold(graph, h.d_hub)]
        used = ip.hbm_in_use()
        for k in range(20):  # nobody holds these: one of a kind at a time
            assert _bins(graph, 4 + k, 200 + k)[0] == 0
            assert _hubs(graph, 300 + k, 128)[0] == 0
        assert ip.hbm_in_use() - used <= (g.V * 4 + 64) + (g.E // 300 + 2) * 16 + (g.E // 128 + g.E // 300 + 8) * 4 + 1024
        assert _bins(graph, 8, 40)[1].d_list[0] == b.d_list[0]
        assert _hubs(graph, 100, 64)[1].d_hub == h.d_hub
        lists = [ip.DeviceArray.wrap(b.d_list[k], b.count[k], np.uint32).to_host() for k in range(3)]
        for k, (lo, hi) in enumerate(((0, 8), (9, 40), (41, 1 << 40))):
            np.testing.assert_array_equal(lists[k], np.flatnonzero((deg >= lo) & (deg <= hi)))
        hub = ip.DeviceArray.wrap(h.d_hub, 4 * h.hubs, np.uint32).to_host().reshape(-1, 4)
        np.testing.assert_array_equal(np.sort(hub[:, 0]), np.flatnonzero(deg > 100))
        with pytest.raises(AssertionError):
            _hold(graph, 16)  # not a set of the graph
        # let go of, a set goes with the next one made
        for p in holds:
            _lib().ipg_hold_release(p)
        used = ip.hbm_in_use()
        assert _bins(graph, 5, 50)[0] == 0
        assert ip.hbm_in_use() < used
        # a hold outlives its graph
        late = _hold(graph, _bins(graph, 5, 50)[1].d_list[0])
    finally:
        graph.free()
    assert ip.hbm_in_use() == base
    _lib().ipg_hold_release(late)
    assert ip.hbm_in_use() == base


def test_held_sets_stay_when_memory_is_short():
    import ipregel_b200 as ip
    g = O.gen_rmat(12, 16, seed=3, undirected=True)
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    holds = []
    try:
        rc, b = _bins(graph, 8, 40)
        rc2, h = _hubs(graph, 100, 64)
        assert rc == 0 and rc2 == 0
        holds = [_hold(graph, b.d_list[0]), _hold(graph, h.d_hub)]
        used = ip.hbm_in_use()
        ip.set_hbm_budget(used + 1024)
        assert _bins(graph, 4, 100)[0] != 0
        assert _hubs(graph, 50, 64)[0] != 0
        assert ip.hbm_in_use() == used
        assert _bins(graph, 8, 40)[1].d_list[0] == b.d_list[0]
        assert _hubs(graph, 100, 64)[1].d_hub == h.d_hub
    finally:
        ip.set_hbm_budget(0)
        for p in holds:
            _lib().ipg_hold_release(p)
        graph.free()


def test_many_users_of_one_graph(monkeypatch):
    """An engine, a server and 18 split plans, each with thresholds of its own: all of them answer bitwise as before the
    others were made, and nothing is left when they are gone."""
    import ipregel_b200 as ip
    from ipregel_b200 import serve as ips
    g = O.gen_rmat(12, 16, seed=5, undirected=True)
    eng = ip.Engine("pagerank", "single_broadcast")
    eng.set_quiet(True)
    eng.release()
    base = ip.hbm_in_use()
    graph = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj)
    plans, srv = [], None
    monkeypatch.setenv("IPG_ORDER", "0")  # the plans on the graph itself, as the engine and the server
    try:
        eng.set_order(False)
        eng.set_param("rounds", 10)
        eng.attach(graph)
        first = eng.run().values.copy()
        srv = ips.Server(ppr_rounds=10)
        gid = srv.add_graph(graph)

        def ask():
            kinds = (ips.PPR, ips.CC)
            ids = [srv.submit(gid, k, 0 if k == ips.CC else 2) for k in kinds]
            srv.drain()
            return [srv.result(q, k, g.V) for q, k in zip(ids, kinds)]

        answers = ask()
        runs = []
        for k in range(18):
            monkeypatch.setenv("IPG_PR_T0", str(2 + k))
            monkeypatch.setenv("IPG_PR_T1", str(70 + k))
            plans.append(ip.PageRankF32(graph))
            runs.append(plans[-1].run(rounds=10)[0].copy())
        np.testing.assert_array_equal(eng.run().values, first)
        for got, want in zip(ask(), answers):
            np.testing.assert_array_equal(got, want)
        for plan, x in zip(plans, runs):
            np.testing.assert_array_equal(plan.run(rounds=10)[0], x)
    finally:
        for plan in plans:
            plan.free()
        if srv is not None:
            srv.free()
        eng.set_order(True)
        eng.release()
        graph.free()
    assert ip.hbm_in_use() == base
