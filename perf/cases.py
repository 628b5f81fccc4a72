"""The work that programs have this engine do, case by case, through its public Python and C entry points.

A case is a dict of plain values; prepare() makes what a program holds before the call (graphs resident on the
GPU, source vertices, result arrays), run() is one pass.  Graphs are the R-MAT (a/b/c = .57/.19/.19, 16 edges per
vertex) and 4-neighbour grid families that the benchmark and the tests use, drawn on the GPU from the seed.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sep-graph_b200"))
import sepgraph as sg  # noqa: E402

EDGE_FACTOR = 16
PR_ERROR = 1e-7
_ctx = None


def context():
    """The program's one context: device, stream and scratch shared by all of its graphs."""
    global _ctx
    if _ctx is None:
        _ctx = sg.Context(0)
    return _ctx


# ---------------------------------------------------------------- cases

def listed():
    return [
        # one BFS of a graph of a thousand vertices: launch and round latency
        {"name": "bfs_small", "kind": "bfs", "nv": 1000},
        # BFS of the benchmark's largest symmetric graph (2^23 vertices, about 250 M edges), default options
        {"name": "bfs_large", "kind": "bfs", "nv": 1 << 23},
        # the headline: weighted R-MAT with 2^22 vertices, near/far delta-stepping as the autotuner picks it
        {"name": "sssp_delta", "kind": "sssp", "nv": 1 << 22, "delta": 8},
        # SSSP with default options (the hybrid policy chooses push or pull per round), ordinary odd size
        {"name": "sssp_hybrid", "kind": "sssp", "nv": 300007, "delta": 0},
        # SSSP on a road-like graph: thousands of small rounds, the autotuner's options for grids
        {"name": "sssp_grid", "kind": "sssp_grid", "rows": 3001, "cols": 2999},
        # PageRank as topology-driven pull, to the benchmark's threshold
        {"name": "pagerank_pull", "kind": "pagerank", "nv": 1 << 22, "variant": "sync_pull_td"},
        # PageRank as data-driven residual push, ordinary odd size
        {"name": "pagerank_push", "kind": "pagerank", "nv": 1000003, "variant": "async_push_dd"},
        # betweenness centrality of one source, forward and backward
        {"name": "bc", "kind": "bc", "nv": 1 << 22},
        # 64 BFS of one graph in one call
        {"name": "msbfs", "kind": "msbfs", "nv": 1 << 22, "nsrc": 64},
        # 32 betweenness sources of one graph in one call, odd size
        {"name": "msbc", "kind": "msbc", "nv": 700001, "nsrc": 32},
        # 256 SSSP queries over nine graphs of 2^12 to 2^20 vertices in one call (a served batch)
        {"name": "sssp_batch", "kind": "sssp_batch", "lo": 12, "hi": 20, "nq": 256},
        # ingest: raw weighted edge list -> cleaned CSR and in-edge view on the device
        {"name": "build", "kind": "build", "nv": 1 << 21, "d2ud": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "sssp", "sssp", "sssp_grid", "pagerank", "pagerank", "bc", "msbfs", "msbfs_grid",
                       "msbc", "sssp_batch", "build"])
    if kind == "bfs":
        return {"kind": kind, "nv": _log_int(rng, 1000, 1 << 23)}
    if kind == "sssp":
        delta = rng.choice([0, 8])
        return {"kind": kind, "nv": _log_int(rng, 1000, 1 << 22 if delta else 400000), "delta": delta}
    if kind == "sssp_grid":
        return {"kind": kind, "rows": _log_int(rng, 50, 3000), "cols": _log_int(rng, 50, 2999)}
    if kind == "pagerank":
        variant = rng.choice(["sync_pull_td", "async_push_dd"])
        return {"kind": kind, "nv": _log_int(rng, 1000, 1 << 22 if variant == "sync_pull_td" else 1 << 20),
                "variant": variant}
    if kind == "bc":
        return {"kind": kind, "nv": _log_int(rng, 1000, 1 << 22)}
    if kind == "msbfs":
        return {"kind": kind, "nv": _log_int(rng, 1000, 1 << 22), "nsrc": rng.randint(8, 64)}
    if kind == "msbfs_grid":
        return {"kind": kind, "rows": _log_int(rng, 50, 1500), "cols": _log_int(rng, 50, 1500),
                "nsrc": rng.randint(8, 64)}
    if kind == "msbc":
        return {"kind": kind, "nv": _log_int(rng, 1000, 700000), "nsrc": rng.randint(8, 32)}
    if kind == "sssp_batch":
        lo = rng.randint(11, 14)
        return {"kind": kind, "lo": lo, "hi": rng.randint(lo + 2, 19), "nq": _log_int(rng, 16, 256)}
    d2ud = rng.random() < 0.4
    return {"kind": kind, "nv": _log_int(rng, 10000, 1 << 20 if d2ud else 1 << 21), "d2ud": d2ud}


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _rmat_edges(nv, gen):
    """EDGE_FACTOR * nv raw R-MAT edges (self-loops and duplicates included), in random order, as int32."""
    scale = max(1, (nv - 1).bit_length())
    m = EDGE_FACTOR * nv
    src = torch.empty(m, dtype=torch.int32, device="cuda")
    dst = torch.empty(m, dtype=torch.int32, device="cuda")
    step = 1 << 25
    for lo in range(0, m, step):
        n = min(step, m - lo)
        u = torch.zeros(n, dtype=torch.int32, device="cuda")
        v = torch.zeros(n, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            r = torch.rand(n, generator=gen, device="cuda")
            bu = r >= 0.76
            bv = ((r >= 0.57) & (r < 0.76)) | (r >= 0.95)
            u = u.mul_(2).add_(bu)
            v = v.mul_(2).add_(bv)
        src[lo:lo + n] = u % nv
        dst[lo:lo + n] = v % nv
    return src, dst


def _grid_csr(rows, cols):
    """CSR of the 4-neighbour grid: up, left, right, down of every vertex, as int32."""
    ids = torch.arange(rows * cols, device="cuda")
    r, c = ids // cols, ids % cols
    have = torch.stack([r > 0, c > 0, c < cols - 1, r < rows - 1], 1)
    to = torch.stack([ids - cols, ids - 1, ids + 1, ids + cols], 1)
    idx = to[have].to(torch.int32)
    off = torch.zeros(rows * cols + 1, dtype=torch.int64, device="cuda")
    off[1:] = have.sum(1).cumsum(0)
    return off.to(torch.int32), idx


def _sources(src, dst, nv, n, gen, symmetric):
    """n vertices with an edge other than a self-loop, uniformly drawn."""
    keep = src != dst
    has = torch.zeros(nv, dtype=torch.bool, device="cuda")
    has[src[keep].long()] = True
    if symmetric:
        has[dst[keep].long()] = True
    ids = has.nonzero().flatten()
    return [int(x) for x in ids[torch.randint(0, len(ids), (n,), generator=gen, device="cuda")]]


def _rmat_graph(nv, gen, symmetric, weights=False, nsrc=1, no_csc=False):
    """(device graph without self-loops and duplicates, nsrc source vertices)."""
    src, dst = _rmat_edges(nv, gen)
    w = torch.randint(1, 64, (len(src),), generator=gen, device="cuda", dtype=torch.int32) if weights else None
    s = _sources(src, dst, nv, nsrc, gen, symmetric)
    torch.cuda.synchronize()
    if symmetric:
        g = context().build_graph(nv, src, dst, w, deself_cycle=True, d2ud=True, no_csc=no_csc)
    else:
        g = context().build_graph(nv, src, dst, w, deself_cycle=True, deduplicate=True, sort_rows=True, no_csc=no_csc)
    return g, s


def prepare(case, seed):
    gen = _generator(seed)
    k = case["kind"]
    st = {"case": case}
    if k == "bfs":
        st["g"], st["src"] = _rmat_graph(case["nv"], gen, True)
        st["out"] = torch.empty(case["nv"], dtype=torch.int32, device="cuda")
    elif k == "sssp":
        st["g"], st["src"] = _rmat_graph(case["nv"], gen, False, weights=True)
        st["out"] = torch.empty(case["nv"], dtype=torch.int32, device="cuda")
    elif k in ("sssp_grid", "msbfs_grid"):
        nv = case["rows"] * case["cols"]
        off, idx = _grid_csr(case["rows"], case["cols"])
        w = torch.randint(1, 1000, (len(idx),), generator=gen, device="cuda", dtype=torch.int32)
        n = case.get("nsrc", 1)
        st["src"] = [int(x) for x in torch.randint(0, nv, (n,), generator=gen, device="cuda")]
        torch.cuda.synchronize()
        if k == "sssp_grid":
            st["g"] = context().graph_from_csr(off, idx, w, no_csc=True)
            st["out"] = torch.empty(nv, dtype=torch.int32, device="cuda")
        else:
            st["g"] = context().graph_from_csr(off, idx, symmetric=True)
            st["out"] = torch.empty((n, nv), dtype=torch.int32, device="cuda")
    elif k == "pagerank":
        st["g"], _ = _rmat_graph(case["nv"], gen, False)
        st["out"] = torch.empty(case["nv"], dtype=torch.float32, device="cuda")
    elif k == "bc":
        st["g"], st["src"] = _rmat_graph(case["nv"], gen, True)
        st["out"] = torch.empty(case["nv"], dtype=torch.float32, device="cuda")
        st["sigma"] = torch.empty(case["nv"], dtype=torch.int64, device="cuda")
    elif k in ("msbfs", "msbc"):
        st["g"], st["src"] = _rmat_graph(case["nv"], gen, True, nsrc=case["nsrc"])
        st["out"] = torch.empty((case["nsrc"], case["nv"]), device="cuda",
                                dtype=torch.int32 if k == "msbfs" else torch.float32)
    elif k == "sssp_batch":
        scales = list(range(case["lo"], case["hi"] + 1))
        per = -(-case["nq"] // len(scales))
        graphs = [_rmat_graph(1 << s, gen, False, weights=True, nsrc=per, no_csc=True) for s in scales]
        st["graphs"] = [g for g, _ in graphs]
        st["queries"], st["outs"], sizes = [], [], []
        for q in range(case["nq"]):
            g, src = graphs[q % len(scales)]
            st["queries"].append((g, src[q // len(scales)]))
            sizes.append(1 << scales[q % len(scales)])
        st["out"] = torch.empty(sum(sizes), dtype=torch.int32, device="cuda")
        st["outs"] = list(st["out"].split(sizes))
    elif k == "build":
        nv = case["nv"]
        st["src"], st["dst"] = _rmat_edges(nv, gen)
        m = len(st["src"])
        st["w"] = torch.randint(1, 64, (m,), generator=gen, device="cuda", dtype=torch.int32)
        cap = 2 * m if case["d2ud"] else m
        # room for every raw edge; what cleaning removes stays zero at the end
        st["csr"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (nv + 1, cap, cap)]
        st["csc"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (nv + 1, cap, cap)]
        context()
        torch.cuda.synchronize()
    else:
        raise ValueError(k)
    return st


# ---------------------------------------------------------------- one pass

def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "bfs":
        return st["g"].bfs(st["src"][0], out=st["out"])[0]
    if k == "sssp":
        if case["delta"]:
            opts = {"variant": "async_push_dd", "priority": "low_high", "priority_delta": case["delta"],
                    "max_iteration": 1000000}
        else:
            opts = {}
        return st["g"].sssp(st["src"][0], out=st["out"], **opts)[0]
    if k == "sssp_grid":
        return st["g"].sssp(st["src"][0], out=st["out"], variant="async_push_dd", priority="low_high",
                            priority_delta=8000, blocks_per_sm=1, worklist=2, local_depth=4, lb_push="fine",
                            max_iteration=10000000)[0]
    if k == "pagerank":
        return st["g"].pagerank(out=st["out"], variant=case["variant"], pr_error=PR_ERROR, max_iteration=100000)[0]
    if k == "bc":
        return st["g"].bc(st["src"][0], out=st["out"], sigma_out=st["sigma"])[:2]
    if k in ("msbfs", "msbfs_grid"):
        return st["g"].msbfs(st["src"], out=st["out"], max_iteration=1000000)[0]
    if k == "msbc":
        return st["g"].msbc(st["src"], out=st["out"])[0]
    if k == "sssp_batch":
        context().sssp_batch(st["queries"], outs=st["outs"], variant="async_push_dd", max_iteration=1000000)
        return st["out"]
    # ingest: build the graph, hand both of its views to the program's own arrays, release it
    flags = {"d2ud": True} if case["d2ud"] else {"deduplicate": True, "sort_rows": True}
    g = context().build_graph(case["nv"], st["src"], st["dst"], st["w"], deself_cycle=True, **flags)
    ne = g.info()["ne"]
    for csc, arrays in ((0, st["csr"]), (1, st["csc"])):
        status = sg.load().sg_graph_copy_out(g.handle, csc, *(a.data_ptr() for a in arrays))
        if status != sg.SG_OK:
            raise RuntimeError(f"sg_graph_copy_out: status {status}")
    g.close()
    return [ne, *st["csr"], *st["csc"]]


# ---------------------------------------------------------------- what a pass cannot do without

def _edges(nv, symmetric):
    """Edges left of the raw R-MAT stream without self-loops and duplicates (fit over 2^10 .. 2^20 vertices)."""
    if symmetric:
        return 2 * EDGE_FACTOR * nv * (1 - 0.36 * (nv / 1024) ** -0.247)
    return EDGE_FACTOR * nv * (1 - 0.27 * (nv / 1024) ** -0.268)


def work(case):
    k = case["kind"]
    nv = case.get("nv") or case.get("rows", 0) * case.get("cols", 0)
    if k == "bfs":
        return {"bytes": 4 * (nv + 1) + 4 * _edges(nv, True) + 4 * nv, "flops": 0}
    if k == "sssp":
        return {"bytes": 4 * (nv + 1) + 8 * _edges(nv, False) + 4 * nv, "flops": 0}
    if k == "sssp_grid":
        return {"bytes": 4 * (nv + 1) + 8 * 4 * nv + 4 * nv, "flops": 0}
    if k == "pagerank":
        # the residual falls by the damping factor per sweep; every sweep reads the edges and the contributions
        # and updates the ranks
        sweeps = math.log(PR_ERROR / 0.15) / math.log(0.85)
        e = _edges(nv, False)
        return {"bytes": sweeps * (4 * (nv + 1) + 4 * e + 12 * nv), "flops": sweeps * 2 * e}
    if k == "bc":
        return {"bytes": 2 * (4 * (nv + 1) + 4 * _edges(nv, True)) + 12 * nv, "flops": 4 * _edges(nv, True)}
    if k == "msbfs":
        return {"bytes": 4 * (nv + 1) + 4 * _edges(nv, True) + 4 * nv * case["nsrc"], "flops": 0}
    if k == "msbfs_grid":
        return {"bytes": 4 * (nv + 1) + 4 * 4 * nv + 4 * nv * case["nsrc"], "flops": 0}
    if k == "msbc":
        e = _edges(nv, True)
        return {"bytes": 2 * (4 * (nv + 1) + 4 * e) + 4 * nv * case["nsrc"], "flops": 4 * e * case["nsrc"]}
    if k == "sssp_batch":
        n = case["hi"] - case["lo"] + 1
        one = [4 * (2 ** s + 1) + 8 * _edges(2 ** s, False) + 4 * 2 ** s for s in range(case["lo"], case["hi"] + 1)]
        return {"bytes": sum(one) * case["nq"] / n, "flops": 0}
    m = EDGE_FACTOR * nv
    e = _edges(nv, case["d2ud"])
    return {"bytes": 12 * m + 2 * (4 * (nv + 1) + 8 * e), "flops": 0}


# ---------------------------------------------------------------- 64-bit results

def _edge_list(nv, src, dst, symmetric):
    """Unique directed edges without self-loops, ordered by (source, destination)."""
    key = torch.unique(src.long()[src != dst] * nv + dst.long()[src != dst])
    if symmetric:
        key = torch.unique(torch.cat([key, key % nv * nv + key // nv]))
    return key // nv, key % nv


def _exact_pagerank(nv, src, dst):
    """Fixed point of p = 0.15 + 0.85 * sum over in-edges of p(u) / outdegree(u)."""
    deg = torch.bincount(src, minlength=nv).double()
    order = torch.argsort(dst, stable=True)
    off = torch.zeros(nv + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(dst, minlength=nv).cumsum(0)
    pull = torch.sparse_csr_tensor(off, src[order], torch.ones(len(src), dtype=torch.float64, device="cuda"),
                                   size=(nv, nv))
    p = torch.full((nv,), 0.15, dtype=torch.float64, device="cuda")
    for _ in range(400):
        q = 0.15 + 0.85 * (pull @ torch.where(deg > 0, p / deg, 0.0))
        change = float((q - p).abs().sum() / q.sum())
        p = q
        if change < 1e-14:
            break
    return p


def _exact_bc(nv, src, dst, source):
    """Brandes' dependency of one source, halved, and 0 at the source."""
    level = torch.full((nv,), -1, dtype=torch.int32, device="cuda")
    sigma = torch.zeros(nv, dtype=torch.float64, device="cuda")
    level[source], sigma[source] = 0, 1
    dag, d = [], 0
    while True:
        out = level[src] == d
        u, v = src[out], dst[out]
        fresh = level[v] < 0
        u, v = u[fresh], v[fresh]
        if not len(u):
            break
        level[v] = d + 1
        sigma.index_add_(0, v, sigma[u])
        dag.append((u, v))
        d += 1
    delta = torch.zeros(nv, dtype=torch.float64, device="cuda")
    for u, v in reversed(dag):
        delta.index_add_(0, u, sigma[u] / sigma[v] * (1 + delta[v]))
    delta[source] = 0
    return delta * 0.5


def exact(case, seed):
    k = case["kind"]
    if k not in ("pagerank", "bc", "msbc"):
        return None  # levels, distances and edge lists are whole numbers
    gen = _generator(seed)
    nv = case["nv"]
    raw = _rmat_edges(nv, gen)
    if k == "pagerank":
        return _exact_pagerank(nv, *_edge_list(nv, *raw, False))
    sources = _sources(*raw, nv, case.get("nsrc", 1), gen, True)
    src, dst = _edge_list(nv, *raw, True)
    del raw
    if k == "bc":
        return _exact_bc(nv, src, dst, sources[0]), None
    return torch.stack([_exact_bc(nv, src, dst, s) for s in sources])
