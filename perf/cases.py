"""Performance cases of the concurrent multi-source BFS.

Each case is one call (or one burst of calls) a user's program makes through
the package's public entry points: ``Graph.run`` on a resident graph, opening
a graph and traversing it, or queries to the serving front-end.  The graphs are
the families and sizes of the benchmark (R-MAT, a Chung-Lu social graph, a
grid) and smaller or ragged ones of the same kinds, generated here on the GPU.

A program keeps one resident graph and traverses it from many source lists,
so the graph (and its server) belongs to the case, ``graph_seed`` included,
and the last one opened stays open; the sources come from the seed.
"""
import random

import numpy as np
import torch

import ibfs_b200 as ib

SOURCE_MAJOR, VERTEX_MAJOR = 0, 1


def _case(name, use="run", graph="rmat", n=128, out="device", width=128, concurrent=0, groupby=0,
          layout=SOURCE_MAJOR, depth_bytes=0, switch_level=-1, graph_seed=1, **shape):
    return dict(name=name, use=use, graph=graph, n=n, out=out, width=width, concurrent=concurrent,
                groupby=groupby, layout=layout, depth_bytes=depth_bytes,
                switch_level=switch_level, graph_seed=graph_seed, **shape)


def listed():
    return [
        # one source on a small graph: launches and barriers, nothing else
        _case("query_small", n=1, scale=12, ef=16, graph_seed=11),
        # one source on the social graph of the serving benchmark: the latency of a lone query
        _case("query_social", graph="social", n=1, V=3_070_000, m=117_000_000, graph_seed=5),
        # the benchmark's smallest batch: R-MAT scale 16, one full batch
        _case("batch_s16", scale=16, ef=16, groupby=1, graph_seed=1),
        # the command line's call: fixed switch level, GroupBy, depths to host memory,
        # several batches with a partial last one, a vertex count that is no multiple of 4
        _case("cli_host_rows", graph="social", n=300, V=200_003, m=3_100_007, out="host",
              groupby=1, switch_level=3, graph_seed=7),
        # the benchmark's ordinary run: R-MAT scale 22, 512 sources in 4 batches
        _case("runs_s22", n=512, scale=22, ef=16, groupby=1, graph_seed=2),
        # the headline: R-MAT scale 24, 1024 sources in 8 batches
        _case("runs_s24", n=1024, scale=24, ef=16, groupby=1, graph_seed=3),
        # the benchmark's high-diameter graph: about 150 small levels per batch
        _case("grid_4096", graph="grid", n=256, rows=4096, cols=4096, shortcuts=0.001,
              depth_bytes=1, graph_seed=4),
        # a road-like strip without shortcuts: over a thousand tiny levels, two-byte depths
        _case("road_deep", graph="grid", n=64, rows=256, cols=1024, shortcuts=0.0, depth_bytes=2,
              graph_seed=9),
        # wide status words and the vertex-major layout on ragged sizes, partial batches
        _case("wide_vertex_major", graph="social", n=700, V=500_009, m=8_000_011, width=256,
              concurrent=250, layout=VERTEX_MAJOR, groupby=2, graph_seed=13),
        # narrow status words: a few sources at a time on a middling graph
        _case("narrow_s20", n=60, scale=20, ef=16, width=32, groupby=2, graph_seed=6),
        # a burst of mixed queries to the server of the serving benchmark's graph
        _case("serve_burst", use="serve", graph="social", n=24, V=3_070_000, m=117_000_000,
              graph_seed=5),
        # a program that opens a graph, traverses one batch and closes it
        _case("open_and_run", use="open", n=128, scale=18, ef=16, groupby=1, graph_seed=8),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    use = rng.choice(["run"] * 7 + ["serve", "open"])
    graph = rng.choice(["rmat", "rmat", "social", "social", "grid"])
    if use == "serve":
        graph = rng.choice(["rmat", "social"])
    shape, depth_bytes = {}, 0
    if graph == "rmat":
        shape = dict(scale=rng.randint(10, 19 if use == "open" else 22), ef=rng.randint(4, 16))
        V = 1 << shape["scale"]
    elif graph == "social":
        V = _log(rng, 2_000, 150_000 if use == "open" else 2_000_000)
        shape = dict(V=V, m=V * rng.randint(4, 24))
    else:
        rows = _log(rng, 32, 256 if use == "open" else 1500)
        cols = _log(rng, 32, 512 if use == "open" else 1500)
        deep = rng.random() < 0.3
        if deep:
            cols = min(cols, 700)
            rows = min(rows, 300)
        shape = dict(rows=rows, cols=cols, shortcuts=0.0 if deep else 0.001)
        V = rows * cols
    if use == "serve":
        n = _log(rng, 1, 24)
    else:
        n = min(_log(rng, 1, 1024), max(1, V // 4), max(1, 1_500_000_000 // V))
    width = rng.choice([32, 64, 128, 128, 128, 256])
    out = "host" if use == "run" and n * V < 100_000_000 and rng.random() < 0.3 else "device"
    if graph == "grid" and out == "device":  # may pass level 254: a host array widens by itself
        depth_bytes = 2
    return dict(use=use, graph=graph, n=n, out=out,
                width=width, concurrent=rng.choice([0, 0, 0, rng.randint(width // 2, width)]),
                groupby=rng.choice([0, 1, 1, 2, 3]) if use != "serve" else 0,
                layout=rng.choice([SOURCE_MAJOR] * 3 + [VERTEX_MAJOR]) if use == "run"
                else SOURCE_MAJOR,
                depth_bytes=depth_bytes,
                switch_level=rng.choice([-1, -1, -1, 3]) if graph != "grid" else -1,
                graph_seed=rng.randint(1, 1 << 20), **shape)


# ---- graphs -----------------------------------------------------------------
def _vertices(c):
    if c["graph"] == "rmat":
        return 1 << c["scale"]
    return c["V"] if c["graph"] == "social" else c["rows"] * c["cols"]


def _edges(c):
    """Undirected edges that the generator draws."""
    if c["graph"] == "rmat":
        return c["ef"] << c["scale"]
    if c["graph"] == "social":
        return c["m"]
    return int(2 * c["rows"] * c["cols"] * 0.95 + c["rows"] * c["cols"] * c["shortcuts"])


def _endpoints(c, gen):
    """(src, dst) of the undirected edges, on the GPU."""
    dev, V, m = "cuda", _vertices(c), _edges(c)
    step = 1 << 24
    if c["graph"] == "rmat":  # a/b/c/d = .57/.19/.19/.05, ids permuted
        perm = torch.randperm(V, device=dev, generator=gen)
        for at in range(0, m, step):
            k = min(step, m - at)
            s = torch.zeros(k, dtype=torch.int64, device=dev)
            d = torch.zeros(k, dtype=torch.int64, device=dev)
            for _ in range(c["scale"]):
                r = torch.rand(k, device=dev, generator=gen)
                s = 2 * s + (r >= 0.76)
                d = 2 * d + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
            yield perm[s], perm[d]
    elif c["graph"] == "social":  # Chung-Lu, exponent 2.1, capped expected degree
        w = torch.arange(1, V + 1, dtype=torch.float64, device=dev).pow(-1.0 / 1.1)
        w = (w * (2.0 * m / w.sum())).clamp(max=33000.0)
        edge = torch.cumsum(w, 0)
        perm = torch.randperm(V, device=dev, generator=gen)
        for at in range(0, m, step):
            r = torch.rand(2, min(step, m - at), dtype=torch.float64, device=dev, generator=gen)
            s, d = torch.searchsorted(edge, r * edge[-1]).clamp_(max=V - 1)
            yield perm[s], perm[d]
    else:  # grid: 5 % of the links deleted, a few random shortcuts
        v = torch.arange(V, device=dev)
        rows, cols = c["rows"], c["cols"]
        for s, d in ((v[v % cols < cols - 1], 1), (v[: (rows - 1) * cols], cols)):
            s = s[torch.rand(s.numel(), device=dev, generator=gen) >= 0.05]
            yield s, s + d
        k = int(V * c["shortcuts"])
        if k:
            s, d = torch.randint(0, V, (2, k), device=dev, generator=gen)
            yield s, d


def _csr(c, seed):
    """Symmetric CSR without loops or duplicates, as host arrays."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    V = _vertices(c)
    keys = []
    for s, d in _endpoints(c, gen):
        keep = s != d
        s, d = s[keep], d[keep]
        keys += [s * V + d, d * V + s]
    keys = torch.cat(keys)
    keys = torch.unique(keys)
    deg = torch.bincount(keys // V, minlength=V)
    beg = torch.zeros(V + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=beg[1:])
    col = (keys % V).to(torch.int32)
    return beg.cpu().numpy(), col.cpu().numpy()


class _Open:
    """The resident graph (and its server) that the program keeps."""

    key = graph = server = busy = None

    @classmethod
    def get(cls, c):
        key = tuple(sorted((k, v) for k, v in c.items()
                           if k in ("graph", "graph_seed", "scale", "ef", "V", "m", "rows", "cols",
                                    "shortcuts")))
        if cls.key != key:
            cls.close()
            beg, col = _csr(c, c["graph_seed"])
            torch.cuda.empty_cache()
            cls.graph = ib.Graph.from_csr(beg, col)
            cls.busy = torch.from_numpy(np.flatnonzero(np.diff(beg)))
            cls.key = key
        return cls

    @classmethod
    def get_server(cls, c):
        key = (c["width"], c["concurrent"])
        if cls.server is None or cls.server[0] != key:
            if cls.server is not None:
                cls.server[1].close()
            cls.server = (key, ib.Server(cls.graph, width=c["width"], concurrent=c["concurrent"],
                                         switch_level=c["switch_level"],
                                         arena_bytes=max(1 << 26, 4096 * cls.graph.V)))
        return cls.server[1]

    @classmethod
    def close(cls):
        if cls.server is not None:
            cls.server[1].close()
        if cls.graph is not None:
            cls.graph.close()
        cls.key = cls.graph = cls.server = cls.busy = None


# ---- the cases --------------------------------------------------------------
def _options(c):
    return dict(width=c["width"], concurrent=c["concurrent"], groupby=c["groupby"],
                depth_bytes=c["depth_bytes"], switch_level=c["switch_level"])


def _query_sizes(c):
    """Sources per query of a burst: 1..256, spread over the logarithm."""
    rng = random.Random(c["graph_seed"])
    return [_log(rng, 1, min(256, _vertices(c) // 4)) for _ in range(c["n"])]


def _sources(busy, n, seed):
    gen = torch.Generator()
    gen.manual_seed(seed)
    at = torch.randint(0, busy.numel(), (n,), generator=gen)
    return busy[at].to(torch.int32).numpy()


def _rows(c, n):
    return torch.empty(n * _vertices(c), device="cuda",
                       dtype=torch.int16 if c["depth_bytes"] == 2 else torch.uint8)


def prepare(case, seed):
    c = case
    if c["use"] == "open":
        beg, col = _csr(c, c["graph_seed"] + 7919 * seed)
        busy = torch.from_numpy(np.flatnonzero(np.diff(beg)))
        return dict(c=c, csr=(beg, col), src=_sources(busy, c["n"], seed), out=_rows(c, c["n"]))
    opened = _Open.get(c)
    if c["use"] == "serve":
        sizes = _query_sizes(c)
        src = _sources(opened.busy, sum(sizes), seed)
        return dict(c=c, server=opened.get_server(c), out=_rows(c, sum(sizes)),
                    queries=np.split(src, np.cumsum(sizes)[:-1]))
    state = dict(c=c, graph=opened.graph, src=_sources(opened.busy, c["n"], seed))
    if c["out"] == "device":
        state["out"] = _rows(c, c["n"])
    return state


def run(state):
    c, out = state["c"], state.get("out")
    if c["use"] == "serve":
        srv, V = state["server"], _vertices(c)
        ids = [(srv.submit(q), len(q)) for q in state["queries"]]
        at = out.data_ptr()
        for qid, k in ids:
            srv.wait(qid, k, out_ptr=at, on_device=True)
            at += k * V
    elif c["use"] == "open":
        with ib.Graph.from_csr(*state["csr"]) as g:
            g.run(state["src"], out_ptr=out.data_ptr(), on_device=True, layout=c["layout"],
                  **_options(c))
    elif c["out"] == "host":
        return state["graph"].run(state["src"], layout=c["layout"], **_options(c)).depth
    else:
        state["graph"].run(state["src"], out_ptr=out.data_ptr(), on_device=True,
                           layout=c["layout"], **_options(c))
    return list(out.chunk(32))


def work(case):
    """The CSR and the sources read once, every depth written once."""
    c = case
    V, n = _vertices(c), c["n"]
    if c["use"] == "serve":
        n = sum(_query_sizes(c))
    return {"bytes": 8.0 * (V + 1) + 8.0 * _edges(c) + 4.0 * n
            + float(n) * V * (2 if c["depth_bytes"] == 2 else 1), "flops": 0.0}


def exact(case, seed):
    """Depths by plain level-synchronous products with the adjacency matrix."""
    c = case
    V, n = _vertices(c), c["n"]
    if (c["use"] != "run" or c["graph"] == "grid" or c["layout"] == VERTEX_MAJOR
            or n * (V + 2.0 * _edges(c)) > 1e9):
        return None
    beg, col = _csr(c, c["graph_seed"])
    busy = torch.from_numpy(np.flatnonzero(np.diff(beg)))
    src = torch.from_numpy(_sources(busy, n, seed)).long().cuda()
    adj = torch.sparse_csr_tensor(torch.from_numpy(beg), torch.from_numpy(col).long(),
                                  torch.ones(len(col), dtype=torch.float64), (V, V),
                                  device="cuda")
    front = torch.zeros(V, n, dtype=torch.float64, device="cuda")
    front[src, torch.arange(n, device="cuda")] = 1.0
    depth = torch.full((V, n), 255, dtype=torch.uint8, device="cuda")
    level = 0
    while bool(front.any()):
        depth[front > 0] = level
        level += 1
        front = ((adj @ front > 0) & (depth == 255)).double()
    if c["out"] == "host":
        return depth.t().contiguous().cpu().numpy()
    return list(depth.t().reshape(-1).chunk(32))
