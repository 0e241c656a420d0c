"""The walks and loads this framework is timed on, each through a public entry point.

A case names the call it makes (`call`), the graph it runs on and the walk:

    host    deepwalk(), node2vec(): a PathSet of host arrays
    into    WalkEngine.walk_into: the paths in the caller's pinned buffers
    device  WalkEngine.walk_device: the packed paths copied into the caller's device tensors
    batch   WalkEngine.batch_walk: many node2vec jobs in one launch
    serve   Server.submit / Server.poll: a burst of node2vec requests
    arrays  WalkEngine.load_arrays of a host CSR, then the first walk on it
    file    WalkEngine.load_graph of a binary edge file, then the first walk on it

With a `scale` the graph is a seeded R-MAT graph (a/b/c = 0.57/0.19/0.19) as in
the benchmark, and the walks start on its vertices that have edges; with
`vertices` it is a random graph of skewed degrees, any vertex count and no
isolated vertex.  weights: 0 none, 1 uniform [1, 5), 2 lognormal(0, 1).  Paths
whose total length depends on the draws (PPR, metapath) go to buffers of the
caller's own, of a fixed size.
"""

import math
import os
import tempfile

import numpy as np
import torch

import knightking_gb300 as kk

SCHEMES = [[1, 2, 4, 8], [2, 8, 2, 16], [4, 1, 16, 4]]


def listed():
    return [
        # an interactive call on a small graph: launches and waits count
        dict(name="deepwalk-small", call="host", app="deepwalk", scale=10, ef=16, weights=2, walkers=1024, length=80),
        # personalised PageRank queries: many walks from a few start vertices
        dict(name="ppr-queries", call="into", app="ppr", scale=18, ef=16, weights=0, walkers=20011, starts=37,
             stop=1.0 / 80),
        # the benchmark's smallest node2vec configuration, a graph that fits L2
        dict(name="node2vec-s16", call="host", app="node2vec", scale=16, ef=16, weights=1, walkers=65536, length=80,
             p=2.0, q=0.5),
        # an odd walker count and length, p and q with the return-edge outlier, into pinned buffers
        dict(name="node2vec-ragged-into", call="into", app="node2vec", scale=19, ef=13, weights=2, walkers=300007,
             length=37, p=0.25, q=3.0),
        # DeepWalk corpus generation: a walker per vertex with edges, alias tables built in the call
        dict(name="deepwalk-s22", call="host", app="deepwalk", scale=22, ef=16, weights=2, walkers=2400000, length=80),
        # PPR over a large unweighted graph, paths consumed on the GPU
        dict(name="ppr-s24-device", call="device", app="ppr", scale=24, ef=16, weights=0, walkers=9000000,
             stop=1.0 / 80),
        # node2vec corpus on a graph far beyond L2, paths consumed on the GPU
        dict(name="node2vec-s22-device", call="device", app="node2vec", scale=22, ef=16, weights=1, walkers=2400000,
             length=80, p=2.0, q=0.5),
        # typed walks with rejection over a large graph
        dict(name="metapath-s22-into", call="into", app="metapath", scale=22, ef=16, weights=1, types=5,
             walkers=2400000, length=80),
        # a batch of uneven node2vec jobs, each with its own p, q, length and walkers
        dict(name="node2vec-batch", call="batch", app="node2vec", vertices=1000003, degree=32, weights=1, jobs=20,
             median=4096),
        # a burst of requests to the server
        dict(name="node2vec-serve", call="serve", app="node2vec", vertices=1000003, degree=32, weights=1, jobs=16,
             median=4096),
        # a graph that is already in host memory, with unsorted adjacencies, and its first walk
        dict(name="arrays-node2vec", call="arrays", app="node2vec", vertices=1000003, degree=24, weights=1,
             walkers=200003, length=40, p=0.5, q=2.0),
        # a graph read from an edge file and made undirected, and its first walk
        dict(name="file-deepwalk", call="file", app="deepwalk", vertices=700001, degree=32, weights=2, walkers=700001,
             length=20),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["host", "host", "into", "device", "device", "batch", "serve", "arrays", "file"])
    pq = dict(p=math.exp(rng.uniform(math.log(0.25), math.log(4.0))),
              q=math.exp(rng.uniform(math.log(0.25), math.log(4.0))))
    if call in ("batch", "serve"):
        return dict(call=call, app="node2vec", vertices=logint(2000, 1000003), degree=rng.randint(6, 32),
                    weights=rng.randint(0, 2), jobs=rng.randint(3, 20), median=logint(64, 8192))
    if call in ("arrays", "file"):
        app = rng.choice(["deepwalk", "node2vec"])
        c = dict(call=call, app=app, vertices=logint(2000, 1000003), degree=rng.randint(6, 32),
                 weights=rng.randint(0, 2), walkers=logint(1000, 500000), length=rng.randint(5, 80))
        return dict(c, **pq) if app == "node2vec" else c
    app = rng.choice(["deepwalk", "node2vec"] if call == "host" else ["deepwalk", "ppr", "node2vec", "metapath"])
    scale = rng.randint(10, 22)
    c = dict(call=call, app=app, scale=scale, ef=rng.randint(8, 16), weights=rng.randint(0, 2),
             walkers=logint(256, 2400000 if scale > 17 else 250000))
    if app == "ppr":
        c["stop"] = 1.0 / rng.randint(10, 100)
        c["starts"] = rng.choice([0, 0, 1, rng.randint(2, 1000)])
    else:
        c["length"] = max(5, min(rng.randint(5, 200), int(2.0e8 / c["walkers"])))
    if app == "node2vec":
        c.update(pq)
    if app == "metapath":
        c["types"] = 5
    return c


def _host_edges(case, seed):
    """Undirected edges (u, v, w) of a random graph: a ring, and endpoints floor(V x^2), so degrees are skewed."""
    V = case["vertices"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed % (1 << 31))
    x = torch.rand(2, V * (case["degree"] - 2) // 2, device="cuda", generator=gen, dtype=torch.float64)
    u, v = (x * x * V).long()
    v = torch.where(u == v, (v + 1) % V, v)
    ring = torch.arange(V, device="cuda")
    u, v = torch.cat([u, ring]), torch.cat([v, (ring + 1) % V])
    order = torch.randperm(len(u), device="cuda", generator=gen)
    u, v = u[order], v[order]
    w = None
    if case["weights"] == 1:
        w = 1.0 + 4.0 * torch.rand(len(u), device="cuda", generator=gen)
    elif case["weights"] == 2:
        w = torch.randn(len(u), device="cuda", generator=gen).exp()
    return u, v, w


def _host_csr(case, seed):
    """Its CSR in host memory: both directions of every edge, neighbours in no order."""
    u, v, w = _host_edges(case, seed)
    V = case["vertices"]
    src, dst = torch.cat([u, v]), torch.cat([v, u])
    order = torch.sort(src, stable=True).indices
    off = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(src, minlength=V).cumsum(0)
    nbr = dst[order].int().cpu().numpy().view(np.uint32)
    return off.cpu().numpy(), nbr, None if w is None else torch.cat([w, w])[order].float().cpu().numpy()


def _requests(case, seed):
    """Requests of the served workload: p, q log-uniform in [1/4, 4], length uniform in [5, 200], walkers lognormal."""
    sizes = np.random.default_rng(1000 * case["median"] + case["jobs"])
    rng = np.random.default_rng(seed)
    reqs = []
    for i in range(case["jobs"]):
        n = int(np.clip(round(sizes.lognormal(math.log(case["median"]), 1.0)), 1, 1 << 17))
        reqs.append(dict(walker_num=n, seed=int(rng.integers(1, 1 << 31)), walk_length=int(sizes.integers(5, 201)),
                         p=float(np.exp(rng.uniform(math.log(0.25), math.log(4.0)))),
                         q=float(np.exp(rng.uniform(math.log(0.25), math.log(4.0)))),
                         walker_begin=int(rng.integers(0, case["vertices"])), weighted=bool(case["weights"])))
    return reqs


class _State:
    """What a user's program holds: the engine, and what the call takes."""

    server = None
    path = None
    starts = None

    def __init__(self, case, seed):
        self.case = case
        self.seed = seed % (1 << 31) + 17

    def __del__(self):
        if self.server is not None:
            self.server.stop()
        if self.path is not None and os.path.exists(self.path):
            os.unlink(self.path)


class _OnDevice:
    """Device memory of an engine as torch sees it; keeps the engine alive."""

    def __init__(self, engine, ptr, count, kind):
        self.engine = engine
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (ptr, False), "version": 3}


def _capacity(case):
    """Vertices the paths take: exactly (length + 1) a walker, or for PPR eight deviations over the mean."""
    n = case["walkers"]
    if case["app"] == "ppr":
        return int((n + 8 * math.sqrt(n)) / case["stop"]) + 1000
    return n * (case["length"] + 1)


def prepare(case, seed):
    s = _State(case, seed)
    call = case["call"]
    s.engine = e = kk.WalkEngine(0)
    if "scale" in case:
        V = 1 << case["scale"]
        e.generate_rmat(case["scale"], case["ef"], seed=seed % (1 << 31) + 1, weights=case["weights"],
                        types=case.get("types", 0))
        # the start vertices: those that have edges, in turn, or a few of them
        length = e.walk_device("deepwalk", V, paths=False, walk_length=1, weighted=False)[1]
        with_edges = (torch.as_tensor(_OnDevice(e, length, V, "<i4"), device="cuda") == 2).nonzero()[:, 0].int()
        if case.get("starts"):
            pick = torch.from_numpy(np.random.default_rng(seed).integers(0, len(with_edges), case["starts"]))
            with_edges = with_edges[pick.cuda()]
        else:
            with_edges = with_edges.repeat(-(-case["walkers"] // len(with_edges)))[:case["walkers"]]
        s.pinned = with_edges.cpu().pin_memory()
        s.starts = s.pinned.numpy().view(np.uint32)
    if call == "into":
        s.length = torch.zeros(case["walkers"], dtype=torch.int32, pin_memory=True)
        s.offset = torch.zeros(case["walkers"], dtype=torch.int64, pin_memory=True)
        s.vertices = torch.zeros(_capacity(case), dtype=torch.int32, pin_memory=True)
    if call == "device":
        s.stream = torch.cuda.Stream()
        e.set_stream(s.stream.cuda_stream)
        s.vertices = torch.zeros(_capacity(case), dtype=torch.int32, device="cuda")
        torch.cuda.current_stream().synchronize()
    if call == "file":
        u, v, w = _host_edges(case, seed)
        cols = [u.int(), v.int()] + ([] if w is None else [w.float().view(torch.int32)])
        fd, s.path = tempfile.mkstemp(suffix=".edges")
        with os.fdopen(fd, "wb") as f:
            f.write(torch.stack(cols, 1).contiguous().cpu().numpy().data)
    if call in ("arrays", "batch", "serve"):
        s.csr = _host_csr(case, seed)
    if call in ("batch", "serve"):
        e.load_arrays(case["vertices"], *s.csr)
        s.csr = None
        s.jobs = _requests(case, seed)
    if call == "serve":
        s.server = e.serve("node2vec", slots=2, max_jobs=64, slot_bytes=1 << 28)
    return s


def _arrays(p):
    return {"length": p.path_length.view(np.int32), "offset": p.offset.view(np.int64),
            "vertices": p.vertices.view(np.int32)}


def _host_walk(s):
    c, e = s.case, s.engine
    kw = dict(seed=s.seed, weighted=bool(c["weights"]), start=s.starts)
    if c["app"] == "deepwalk":
        return _arrays(kk.deepwalk(e, c["walkers"], c["length"], **kw))
    return _arrays(kk.node2vec(e, kk.Node2vecConf(c["p"], c["q"], c["walkers"], c["length"]), **kw))


def _walk_kw(s):
    c = s.case
    kw = dict(seed=s.seed, weighted=bool(c["weights"]), start=s.starts)
    if c["app"] == "ppr":
        return dict(kw, terminate_prob=c["stop"])
    kw["walk_length"] = c["length"]
    if c["app"] == "node2vec":
        kw.update(p=c["p"], q=c["q"])
    if c["app"] == "metapath":
        kw.update(schemes=SCHEMES, scheme_round_robin=True)
    return kw


def run(state):
    s, c, e = state, state.case, state.engine
    call, n = c["call"], c.get("walkers")
    if call == "into":
        e.walk_into(c["app"], n, s.length.data_ptr(), s.offset.data_ptr(), s.vertices.data_ptr(), len(s.vertices),
                    **_walk_kw(s))
        return {"length": s.length, "offset": s.offset, "vertices": s.vertices}
    if call == "device":
        steps, length, offset, vertices = e.walk_device(c["app"], n, **_walk_kw(s))
        # the engine's buffers are the next walk's too: a consumer takes the paths into its own
        with torch.cuda.stream(s.stream):
            s.vertices[:steps + n].copy_(torch.as_tensor(_OnDevice(e, vertices, steps + n, "<i4"), device="cuda"))
        return {"length": torch.as_tensor(_OnDevice(e, length, n, "<i4"), device="cuda"),
                "offset": torch.as_tensor(_OnDevice(e, offset, n, "<i8"), device="cuda"), "vertices": s.vertices}
    if call == "batch":
        return [_arrays(p) for p in e.batch_walk("node2vec", s.jobs)]
    if call == "serve":
        tickets = [s.server.submit(**job) for job in s.jobs]
        return [_arrays(s.server.poll(t).paths) for t in tickets]
    if call == "arrays":
        e.load_arrays(c["vertices"], *s.csr)
    elif call == "file":
        e.load_graph(c["vertices"], s.path, load_as_undirected=True, kind="f32" if c["weights"] else "unweighted")
    return _host_walk(s)


def work(case):
    """Bytes of the graph's parts the call reads, once, and of the paths it writes; flops: none to speak of."""
    c = case
    if "scale" in c:
        V = 1 << c["scale"]
        # measured on R-MAT: the share of the drawn edges left after duplicates
        E = 2 * c["ef"] * V * (1.0 - 0.044 * 2.0 ** ((22 - c["scale"]) / 4.5))
    else:
        V = c["vertices"]
        E = c["degree"] * V
    graph = 8.0 * V + E * (4 + (4 if c["weights"] else 0) + (1 if c.get("types") else 0))
    if c["call"] in ("batch", "serve"):
        walkers = c["jobs"] * c["median"] * math.exp(0.5)
        steps = walkers * 102
    else:
        walkers = c["walkers"]
        if c["app"] == "ppr":
            steps = walkers * (1.0 / c["stop"] - 1)
        elif c["app"] == "metapath":
            steps = walkers * min(16.0, c["length"])  # most walks end where no edge has the wanted type
        else:
            steps = walkers * c["length"]
    if not c["weights"] and c["call"] not in ("arrays", "file"):
        graph = min(graph, 4.0 * steps)  # no tables: only what the walks touch
    return {"bytes": graph + 4.0 * (steps + walkers) + 12.0 * walkers, "flops": 0}


def exact(case, seed):
    """Paths are whole numbers: nothing here is computed in floating point."""
    return None
