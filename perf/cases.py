"""Cases for timing the framework's paths over their real range.

A case is one call a user makes on a graph that is already resident in HBM:

  engine   one program in one version, as run_app does it (parameters, attach, run), the values read on the device
  f32      PageRank's precision split (FP32 values, compensated gathers) from its plan
  batch    connected components and weighted shortest paths over many small graphs in one fused launch
  serve    a mix of queries answered together by the request server

The graphs are synthetic with the shapes of the benchmark and the tests: R-MAT (a/b/c = 0.57/0.19/0.19, self-loops and
duplicate edges removed) with its heavy-tailed degrees, and Erdos-Renyi.  `n` is the number of vertices (any number, not
only powers of two) and `m` the number of sampled edges; undirected graphs hold every edge in both directions.
"""
import ctypes
import math

import numpy as np
import torch

import ipregel_b200 as ip
from ipregel_b200 import batch as ipb
from ipregel_b200 import serve as ips

RMAT_A, RMAT_B, RMAT_C = 0.57, 0.19, 0.19
DAMPING = 0.85


def engine(name, app, version, kind, n, m, undirected, rounds=0, id_bits=32, wmax=0):
    return {"name": name, "path": "engine", "app": app, "version": version, "kind": kind, "n": n, "m": m,
            "undirected": undirected, "rounds": rounds, "id_bits": id_bits, "wmax": wmax}


def listed():
    return [
        # The headline workload: both programs on the undirected scale-24 graph with weights.
        engine("cc_rmat24", "cc", "spread", "rmat", 1 << 24, 16 << 24, True),
        engine("sssp_weighted_rmat24", "sssp_weighted", "spread", "rmat", 1 << 24, 16 << 24, True, wmax=255),
        # PageRank at its largest: 30 rounds in FP64 and with the precision split, directed scale 25.
        engine("pagerank_rmat25", "pagerank", "single_broadcast", "rmat", 1 << 25, 16 << 25, False, rounds=30),
        {"name": "pagerank_f32_rmat25", "path": "f32", "kind": "rmat", "n": 1 << 25, "m": 16 << 25,
         "undirected": False, "rounds": 30, "compensated": True},
        # The plain PageRank configuration: scale 16, 10 rounds; launches and latency count.
        engine("pagerank_rmat16", "pagerank", "single_broadcast", "rmat", 1 << 16, 16 << 16, False, rounds=10),
        # A personalised PageRank query as the plain program answers it.
        engine("ppr_rmat22", "ppr", "single_broadcast", "rmat", 3_999_971, 16 << 22, True, rounds=20),
        # The other two versions of the engine at the size that the reference's makefile targets are compared at.
        engine("cc_combiner_rmat20", "cc", "combiner", "rmat", 1 << 20, 16 << 20, True),
        engine("sssp_hops_spread_pull_rmat20", "sssp", "single_broadcast_spread", "rmat", 1 << 20, 16 << 20, True),
        # 64-bit ids, a flat degree distribution and an odd size.
        engine("cc64_er", "cc", "spread", "er", 1_000_003, 8_000_024, True, id_bits=64),
        # The smallest call: nothing but launches.
        engine("cc_rmat10", "cc", "spread", "rmat", 1 << 10, 16 << 10, True),
        # Many small graphs in one launch, with the push/pull switch that the autotuner offers.
        {"name": "batch_er256", "path": "batch", "parts": 256, "lo": 1024, "hi": 65536, "degree": 8, "wmax": 64,
         "pull_div": 20},
        # Queries of the serving mix (60 % SSSP, 30 % PPR, 10 % CC) that meet on one graph.
        {"name": "serve_rmat20", "path": "serve", "kind": "rmat", "n": 1 << 20, "m": 16 << 20, "undirected": True,
         "wmax": 255, "sssp": 14, "ppr": 7, "cc": 3, "rounds": 20},
    ]


# (app, version, id widths, rounds of rank programs, needs weights): what draw() picks from.
PROGRAMS = (
    ("cc", "spread", (32, 64), 0, False), ("cc", "combiner", (32, 64), 0, False),
    ("cc", "single_broadcast", (32, 64), 0, False), ("cc", "single_broadcast_spread", (32, 64), 0, False),
    ("sssp", "spread", (32, 64), 0, False), ("sssp", "single_broadcast_spread", (32, 64), 0, False),
    ("sssp_weighted", "spread", (32,), 0, True), ("sssp_weighted", "combiner", (32,), 0, True),
    ("pagerank", "single_broadcast", (32,), 30, False), ("pagerank", "combiner", (32,), 10, False),
    ("ppr", "single_broadcast", (32,), 20, False),
)


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(("engine", "f32", "batch", "serve"), (7, 2, 1, 2))[0]
    if path == "batch":
        return {"path": "batch", "parts": _log_uniform(rng, 8, 256), "lo": 1024, "hi": 65536, "degree": 8,
                "wmax": 64, "pull_div": rng.choice((0, 4, 20))}
    kind = rng.choice(("rmat", "rmat", "er"))
    undirected = rng.random() < 0.6
    if path == "serve":
        n = _log_uniform(rng, 1 << 12, 1 << 21)
        return {"path": "serve", "kind": kind, "n": n, "m": n * rng.randint(6, 16), "undirected": undirected,
                "wmax": 255, "sssp": rng.randint(1, 24), "ppr": rng.randint(1, 12), "cc": rng.randint(0, 3),
                "rounds": 20}
    n = _log_uniform(rng, 1 << 10, 1 << 24)
    m = n * rng.randint(5, 16)
    if path == "f32":
        return {"path": "f32", "kind": kind, "n": n, "m": m, "undirected": undirected, "rounds": rng.randint(5, 30),
                "compensated": rng.random() < 0.8}
    app, version, widths, rounds, weighted = rng.choice(PROGRAMS)
    c = engine("", app, version, kind, n, m, undirected, rounds=rounds, id_bits=rng.choice(widths),
               wmax=255 if weighted else 0)
    del c["name"]
    return c


# ---- inputs ----------------------------------------------------------------

def _sample(kind, n, m, gen):
    """m sampled edges (source, target), int32 each."""
    dev = "cuda"
    if kind == "er":
        return (torch.randint(0, n, (m,), generator=gen, device=dev, dtype=torch.int32),
                torch.randint(0, n, (m,), generator=gen, device=dev, dtype=torch.int32))
    levels = max(1, (n - 1).bit_length())
    s = torch.zeros(m, dtype=torch.int32, device=dev)
    d = torch.zeros(m, dtype=torch.int32, device=dev)
    r = torch.empty(m, dtype=torch.float32, device=dev)
    for _ in range(levels):
        r.uniform_(0, 1, generator=gen)
        low = r >= RMAT_A + RMAT_B
        s.mul_(2).add_(low)
        d.mul_(2).add_(((r >= RMAT_A) & ~low) | (r >= RMAT_A + RMAT_B + RMAT_C))
    if n != 1 << levels:  # the vertex ids spread evenly over [0, n), their order kept
        s = ((s.to(torch.int64) * n) >> levels).to(torch.int32)
        d = ((d.to(torch.int64) * n) >> levels).to(torch.int32)
    return s, d


def _csr(kind, n, m, undirected, wmax, seed, id_bits=32):
    """(row starts int64[n + 1], neighbour ids, weights or None) of a graph without self-loops or duplicate edges."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 2_654_435_761 % (1 << 62) + 1)
    s, d = _sample(kind, n, m, gen)
    keep = s != d
    s, d = s[keep], d[keep]
    del keep
    keys = s.to(torch.int64) * n + d
    if undirected:
        keys = torch.cat((keys, d.to(torch.int64) * n + s))
    del s, d
    keys = torch.unique(keys)
    row = torch.searchsorted(keys, torch.arange(n + 1, dtype=torch.int64, device="cuda") * n)
    src = torch.div(keys, n, rounding_mode="floor")
    dst = keys - src * n
    del keys
    wgt = None
    if wmax:
        h = torch.minimum(src, dst) * 2_654_435_761 + torch.maximum(src, dst) * 40_503 + int(seed) % 65_521
        h = (h ^ (h >> 15)) * 2_246_822_519
        wgt = (((h >> 17) & 0x7FFFFFFF) % wmax + 1).to(torch.int32)
        del h
    adj = dst if id_bits == 64 else dst.to(torch.int32)
    return row, adj.contiguous(), wgt


def _resident(n, csr, directed, symmetric, id_bits=32):
    """A Graph over buffers already on the device."""
    row, adj, wgt = csr
    torch.cuda.synchronize()
    h = ctypes.c_void_p()
    E = adj.numel()
    rc = ip.runtime().ipg_graph_from_device(n, E, row.data_ptr(), adj.data_ptr() if E else None, id_bits // 8,
                                            wgt.data_ptr() if wgt is not None and E else None,
                                            4 if wgt is not None else 0, int(directed), 0, ctypes.byref(h))
    if rc != 0:
        raise ip.IPregelError(ip.runtime().ipg_last_error().decode())
    g = ip.Graph(h.value)
    if symmetric:
        g.set_symmetric(True)
    return g


class _View:
    """Device memory of the framework as torch sees it."""

    def __init__(self, ptr, n, typestr, owner):
        self.owner = owner  # kept as long as the tensor
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _tensor(ptr, n, typestr, owner):
    return torch.as_tensor(_View(ptr, n, typestr, owner), device="cuda")


def _graph(case, seed):
    csr = _csr(case["kind"], case["n"], case["m"], case["undirected"], case.get("wmax", 0), seed,
               case.get("id_bits", 32))
    # directed = False, as the reference's benchmarks load their graphs: the stored rows are the gather lists
    return csr, _resident(case["n"], csr, False, case["undirected"], case.get("id_bits", 32))


def prepare(case, seed):
    state = {"case": case}
    if case["path"] == "batch":
        rng = np.random.Generator(np.random.PCG64(case["parts"]))  # the sizes are the case's, the edges the seed's
        sizes = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["parts"])).astype(np.int64)
        state["csr"] = [_csr("er", int(n), int(n) * case["degree"], False, case["wmax"], int(seed) * 1000 + i)
                        for i, n in enumerate(sizes)]
        parts = [_resident(int(n), c, True, False) for n, c in zip(sizes, state["csr"])]
        state["batch"] = ipb.Batch(parts)
        state["runner"] = r = ipb.BatchRunner(state["batch"])
        for k in r.tuning:
            r.tuning[k]["pull_div"] = case["pull_div"]
        torch.cuda.empty_cache()
        return state
    state["csr"], g = _graph(case, seed)
    state["graph"] = g
    if case["path"] == "engine":
        state["engine"] = eng = ip.Engine(case["app"], case["version"], case["id_bits"])
        eng.set_quiet()
        eng.set_tuning()
        if case["app"] == "sssp_weighted":
            eng.set_param_ptr("batch_offsets", None, 0)
        state["params"] = {"rounds": case["rounds"]} if case["rounds"] else {}
        if case["app"] not in ("cc", "pagerank"):
            state["params"]["source"] = 0
    elif case["path"] == "f32":
        state["plan"] = ip.PageRankF32(g)
        state["x"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
        state["diag"] = torch.empty((case["rounds"] + 1, 3), dtype=torch.float64, device="cuda")
    else:
        srv = ips.Server(ppr_rounds=case["rounds"])
        gid = srv.add_graph(g)
        for kind, _ in _queries(case, seed):
            srv.reserve(gid, kind)
        state.update(server=srv, gid=gid, queries=_queries(case, seed), done=[])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the sampling's temporaries go back to the device
    return state


def _queries(case, seed):
    """(kind, source) in order of arrival; uniformly random sources, as the serving trace has them."""
    kinds = [ips.SSSP] * case["sssp"] + [ips.PPR] * case["ppr"] + [ips.CC] * case["cc"]
    kinds = [kinds[i] for i in np.random.Generator(np.random.PCG64(len(kinds))).permutation(len(kinds))]
    rng = np.random.Generator(np.random.PCG64(int(seed) + 77))
    return [(k, 0 if k == ips.CC else int(rng.integers(0, case["n"]))) for k in kinds]


# ---- one pass --------------------------------------------------------------

def _values(eng, V):
    p = ctypes.c_void_p()
    if eng.lib.ipg_app_values_device(ctypes.byref(p)) != 0:
        raise ip.IPregelError(eng.lib.ipg_app_last_error().decode())
    dt = eng.value_dtype
    return _tensor(p.value, V, ("<f" if dt.kind == "f" else "<i") + str(dt.itemsize), eng)


def run(state):
    case = state["case"]
    if case["path"] == "engine":
        eng = state["engine"]
        for k, v in state["params"].items():
            eng.set_param(k, v)
        eng.attach(state["graph"])
        eng.run_only()
        return {"values": _values(eng, case["n"]), "counts": np.array(eng.counts(), dtype=np.int64)}
    if case["path"] == "f32":
        x, diag = state["x"], state["diag"]
        state["plan"].run_device(_Out(x, np.float32), _Out(diag, np.float64), case["rounds"], DAMPING,
                                 case["compensated"], torch.cuda.current_stream().cuda_stream)
        return {"values": x, "diag": diag}
    if case["path"] == "batch":
        r, V = state["runner"], state["batch"].union.V
        r.prepare()
        r.run()
        return {"cc": _values(r.cc, V), "sssp": _values(r.sp, V)}
    srv = state["server"]
    for q in state["done"]:  # the last pass's results
        srv.release(q)
    state["done"] = qids = [srv.submit(state["gid"], k, s) for k, s in state["queries"]]
    srv.drain()
    out = []
    for q, (kind, _) in zip(qids, state["queries"]):
        p, b = ctypes.c_void_p(), ctypes.c_uint64()
        if ip.runtime().ipg_server_result_device(srv._p, q, ctypes.byref(p), ctypes.byref(b)) != 0:
            raise ip.IPregelError(ip.runtime().ipg_last_error().decode())
        out.append(_tensor(p.value, case["n"], "<f4" if kind == ips.PPR else "<i4", srv))
    return out


class _Out:
    """A torch tensor in the place of a DeviceArray."""

    def __init__(self, t, dtype):
        self.ptr, self.n, self.dtype = t.data_ptr(), t.numel(), np.dtype(dtype)


# ---- work and exact results ------------------------------------------------

def work(case):
    if case["path"] == "batch":
        n = int(case["parts"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]))
        e = n * case["degree"]
        return {"bytes": 2 * (8 * n + 4 * e) + 4 * e + 8 * n, "flops": 0}
    n, e = case["n"], case["m"] * (2 if case["undirected"] else 1)
    ids = case.get("id_bits", 32) // 8
    if case["path"] == "serve":
        # the min-plus queries together and the rank queries together read the graph once a superstep at least
        return {"bytes": (case["rounds"] + 1) * (8 * n + 4 * e) + 4 * e + 4 * n * (case["sssp"] + case["ppr"] + case["cc"]),
                "flops": 2 * e * case["rounds"] * case["ppr"]}
    if case["path"] == "f32":
        return {"bytes": case["rounds"] * (8 * n + 4 * e + 8 * n), "flops": 2 * e * case["rounds"]}
    if case["rounds"]:
        return {"bytes": case["rounds"] * (8 * n + ids * e + 16 * n), "flops": 2 * e * case["rounds"]}
    return {"bytes": 8 * n + ids * e + (4 * e if case["wmax"] else 0) + ids * n, "flops": 0}


def _ranks(row, adj, n, rounds, seed_vertex=None, push=False):
    """Yields the FP64 ranks of every superstep (0 .. rounds).  The rows are the gather lists, or (push) the lists that
    shares go out along."""
    deg = (row[1:] - row[:-1]).to(torch.float64)
    if push:
        count = row[1:] - row[:-1]

        def received(b):
            return torch.zeros_like(b).index_add_(0, adj, b.repeat_interleave(count))
    else:
        a = torch.sparse_csr_tensor(row.to(torch.int32), adj, torch.ones(adj.numel(), dtype=torch.float64, device="cuda"),
                                    size=(n, n), check_invariants=False)

        def received(b):
            return torch.mv(a, b)
    if seed_vertex is None:
        x = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        tele = (1.0 - DAMPING) / n
    else:
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        x[seed_vertex] = 1.0
        tele = x * (1.0 - DAMPING)
    yield x
    for _ in range(rounds):
        b = torch.where(deg > 0, x / deg.clamp(min=1), torch.zeros_like(x))
        x = tele + DAMPING * received(b)
        yield x


def exact(case, seed):
    if case["path"] == "batch" or (case["path"] == "engine" and not case["rounds"]):
        return None  # whole numbers
    row, adj, _ = _csr(case["kind"], case["n"], case["m"], case["undirected"], case.get("wmax", 0), seed)
    n = case["n"]
    if case["path"] == "engine":
        x = None
        for x in _ranks(row, adj, n, case["rounds"], 0 if case["app"] == "ppr" else None,
                        push=case["version"] == "combiner"):
            pass
        return {"values": x, "counts": None}
    if case["path"] == "f32":
        diag, prev, x = [], None, None
        empty = row[1:] == row[:-1]
        for x in _ranks(row, adj, n, case["rounds"]):
            moved = torch.zeros((), dtype=torch.float64, device="cuda") if prev is None else (x - prev).abs().sum()
            diag.append(torch.stack((x.sum(), x[empty].sum(), moved)))
            prev = x
        return {"values": x, "diag": torch.stack(diag)}
    out = []
    for kind, source in _queries(case, seed):
        x = None
        if kind == ips.PPR:
            for x in _ranks(row, adj, n, case["rounds"], source):
                pass
        out.append(x)
    return out
