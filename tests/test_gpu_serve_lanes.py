"""The server's gathers at their edges: numbers of lanes around the quads a superstep walks, rows around the thread,
stream and hub-chunk classes (256 edges), and lanes that leave while others gather and join again later."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

PPR_TOL = 2e-6  # FP32 lanes against the FP64 oracle, max abs per vertex
# around four ids (4), 32 edges of a stream, the classes (8, 64, 256) and hub chunks of 256 edges
LENGTHS = (1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025,
           1537, 4095, 4096, 4097, 4609)


def _graph():
    """Symmetric: vertex i < len(LENGTHS) has LENGTHS[i] neighbours among the others; the last 50 vertices none."""
    rng = np.random.default_rng(5)
    V, H = 6000, len(LENGTHS)
    a = np.concatenate([np.full(d, i) for i, d in enumerate(LENGTHS)])
    b = np.concatenate([rng.choice(V - H - 50, d, replace=False) + H for d in LENGTHS])
    src, dst = np.concatenate((a, b)), np.concatenate((b, a))
    order = np.argsort(src, kind="stable")
    src, dst = src[order], dst[order]
    deg = np.bincount(src, minlength=V)
    idx = np.concatenate(([0], np.cumsum(deg)[:-1])).astype(np.uint64)
    return O.add_weights(O.CSR(V, int(deg.sum()), idx, dst.astype(np.uint32), None), wmax=255, seed=5)


@pytest.fixture(scope="module")
def ppr_case():
    g = _graph()
    srcs = [int(s) for s in np.random.default_rng(9).choice(np.flatnonzero(np.diff(g.idx.astype(np.int64), append=g.E)),
                                                            40, replace=False)]
    srcs[1] = len(LENGTHS) - 1  # a hub, and a vertex without neighbours
    srcs[2] = g.V - 1
    return g, srcs, [O.run(g, "ppr", "single_broadcast", source=s, rounds=20)[0] for s in srcs]


@pytest.mark.parametrize("first,later", [(1, 3), (3, 2), (4, 1), (5, 3), (7, 9), (8, 1), (9, 8), (16, 1), (17, 15), (32, 8)])
def test_ppr_lanes_around_the_quads(ppr_case, first, later):
    """`first` queries, `later` more after some supersteps, and when all have left a last one."""
    import ipregel_b200 as ip
    from ipregel_b200 import serve as S
    g, srcs, want = ppr_case
    d = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj, wgt=g.wgt)
    srv = S.Server(ppr_rounds=20)
    try:
        gid = srv.add_graph(d)
        ids = [srv.submit(gid, S.PPR, s) for s in srcs[:first]]
        while srv.stats()["supersteps"] < 7:
            srv.poll()
        ids += [srv.submit(gid, S.PPR, s) for s in srcs[first:first + later]]
        srv.drain()
        ids.append(srv.submit(gid, S.PPR, srcs[0]))
        srv.drain()
        got = [srv.result(q, S.PPR, g.V) for q in ids]
        for x, w in zip(got, want[:first + later] + want[:1]):
            assert np.max(np.abs(x.astype(np.float64) - w)) <= PPR_TOL
        np.testing.assert_array_equal(got[-1].view(np.uint32), got[0].view(np.uint32))
    finally:
        srv.free()
        d.free()


@pytest.fixture(scope="module")
def sssp_case():
    g = _graph()
    srcs = [int(s) for s in np.random.default_rng(10).choice(np.flatnonzero(np.diff(g.idx.astype(np.int64), append=g.E)),
                                                             66, replace=False)]
    srcs[1] = len(LENGTHS) - 1
    srcs[2] = g.V - 1
    return g, srcs, [O.dijkstra(g, s) for s in srcs], O.run(g, "cc", "spread")[0]


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("first,later", [(1, 1), (4, 3), (5, 4), (8, 1), (9, 8), (16, 1), (17, 16), (33, 3), (40, 2), (64, 2)])
def test_sssp_lanes_around_the_quads(sssp_case, symmetric, first, later):
    """`first` queries, `later` more after two supersteps, and a last one on cleared lanes; components beside them
    (union-find on the symmetric graph, a label lane on the other)."""
    import ipregel_b200 as ip
    from ipregel_b200 import serve as S
    g, srcs, want, comp = sssp_case
    d = ip.Graph.from_csr(g.V, g.E, g.idx, g.adj, wgt=g.wgt)
    d.set_symmetric(symmetric)
    srv = S.Server()
    try:
        gid = srv.add_graph(d)
        ids = [srv.submit(gid, S.SSSP, s) for s in srcs[:first]]
        while srv.stats()["supersteps"] < 2:
            srv.poll()
        ids += [srv.submit(gid, S.SSSP, s) for s in srcs[first:first + later]]
        cc = srv.submit(gid, S.CC, 0)
        srv.drain()
        ids.append(srv.submit(gid, S.SSSP, srcs[0]))
        srv.drain()
        for q, w in zip(ids, want[:first + later] + want[:1]):
            np.testing.assert_array_equal(srv.result(q, S.SSSP, g.V), w)
        np.testing.assert_array_equal(srv.result(cc, S.CC, g.V), comp)
    finally:
        srv.free()
        d.free()
