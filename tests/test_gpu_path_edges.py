"""The launch paths at the sizes where they change: hubs around the split
thresholds of pull and backward passes, tiles with their last edge on and off
a boundary and with few or many rows, radix passes around a tile and a digit,
levels past the multi-source bit planes.  Against the oracle; whole numbers
exactly, PageRank L1 <= 1e-6 (normalised, FP64 fixed point), BC 1e-4 relative
+ 1e-5 absolute as in the parity tests."""
import numpy as np
import pytest

import oracle
import sepgraph as sg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sg.Context(0)
    yield c
    c.close()


def _csr(nv, s, d, w=None):
    o = np.argsort(s, kind="stable")
    off = np.zeros(nv + 1, np.uint32)
    off[1:] = np.cumsum(np.bincount(s, minlength=nv))
    return off, np.ascontiguousarray(d[o], np.uint32), None if w is None else np.ascontiguousarray(w[o], np.uint32)


def _hub(k, tail=7):
    """Vertex 0 -> k spokes -> one hub -> a chain; the hub has k in-edges (and, reversed, k out-edges)."""
    spokes = np.arange(1, k + 1, dtype=np.uint32)
    hub = k + 1
    chain = np.arange(hub, hub + tail, dtype=np.uint32)
    s = np.concatenate([np.zeros(k, np.uint32), spokes, chain])
    d = np.concatenate([spokes, np.full(k, hub, np.uint32), chain + 1])
    return hub + tail + 1, s, d


# in-degrees around the warp threshold (32), a tile (256), the split threshold (512) and several chunks
HUBS = [31, 32, 33, 255, 256, 257, 511, 512, 513, 1300, 5000]


@pytest.mark.parametrize("k", HUBS)
@pytest.mark.parametrize("variant", ["async_pull_dd", "sync_pull_dd", "auto"])
def test_pull_into_hub(ctx, k, variant):
    nv, s, d = _hub(k)
    off, idx, _ = _csr(nv, s, d)
    G = ctx.graph_from_csr(off, idx)
    assert np.array_equal(G.bfs(0, variant=variant)[0], oracle.bfs(off, idx, 0))
    G.close()
    w = np.random.default_rng(k).integers(1, 64, len(s)).astype(np.uint32)
    off, idx, w = _csr(nv, s, d, w)
    G = ctx.graph_from_csr(off, idx, w)
    assert np.array_equal(G.sssp(0, variant=variant)[0], oracle.sssp(off, idx, w, 0))
    G.close()


@pytest.mark.parametrize("k", HUBS)
@pytest.mark.parametrize("variant", ["async_pull_dd", "async_push_dd", "auto"])
@pytest.mark.parametrize("back", [False, True])
def test_bc_hub(ctx, k, variant, back):
    nv, s, d = _hub(k)
    if back:  # the hub's k edges lead out: the backward pass sums over them
        s, d = np.concatenate([s, d]), np.concatenate([d, s])
    off, idx, _ = _csr(nv, s, d)
    src = nv - 1 if back else 0
    G = ctx.graph_from_csr(off, idx)
    bc, sigma, _ = G.bc(src, variant=variant)
    want, sig, _ = oracle.bc_f64(off, idx, src)
    assert np.array_equal(sigma.astype(np.float64), sig)
    assert np.all(np.abs(bc - want) <= 1e-4 * np.abs(want) + 1e-5)
    bc2 = ctx.bc_batch([(G, src), (G, 0)], variant=variant)[0][0]
    assert np.all(np.abs(bc2 - want) <= 1e-4 * np.abs(want) + 1e-5)
    G.close()


@pytest.mark.parametrize("k", [1, 33, 513, 5000])
@pytest.mark.parametrize("opts", [{"worklist": 2}, {"worklist": 1}, {"wl_sort": True}])
def test_bc_level_stack_by_worklist(ctx, k, opts):
    """Path counts and dependencies do not depend on how the rounds keep their worklists."""
    nv, s, d = _hub(k)
    off, idx, _ = _csr(nv, np.concatenate([s, d]), np.concatenate([d, s]))
    G = ctx.graph_from_csr(off, idx)
    queries = [(G, 0), (G, nv - 1), (G, 1)]
    out = ctx.bc_batch(queries, variant="async_push_dd", lb_push="fine", **opts)[0]
    for q, (_, src) in enumerate(queries):
        want, sig, _ = oracle.bc_f64(off, idx, src)
        bc, sigma, _ = G.bc(src, variant="async_push_dd", lb_push="fine", **opts)
        assert np.array_equal(sigma.astype(np.float64), sig)
        assert np.all(np.abs(bc - want) <= 1e-4 * np.abs(want) + 1e-5)
        assert np.all(np.abs(out[q] - want) <= 1e-4 * np.abs(want) + 1e-5)
    G.close()


def _random(nv, m, seed, lo=0):
    r = np.random.default_rng(seed)
    return r.integers(lo, nv, m).astype(np.uint32), r.integers(lo, nv, m).astype(np.uint32)


# edges around the 256-edge tile; vertices from one row per tile to a row per edge and mostly empty rows
TILES = [(1, 3), (2, 255), (5, 256), (40, 257), (95, 512), (97, 513), (300, 511), (1000, 1024), (3000, 2049), (9000, 300)]


@pytest.mark.parametrize("nv,m", TILES)
@pytest.mark.parametrize("variant", ["async_pull_dd", "sync_pull_dd", "sync_pull_td", "auto"])
def test_sssp_relax_tiles(ctx, nv, m, variant):
    s, d = _random(nv, m, nv + m)
    off, idx, w = _csr(nv, s, d, np.random.default_rng(m).integers(0, 1000, m).astype(np.uint32))
    G = ctx.graph_from_csr(off, idx, w)
    src = int(s[0])
    want = oracle.sssp(off, idx, w, src)
    assert np.array_equal(G.sssp(src, variant=variant, max_iteration=100000)[0], want)
    other = (src + nv // 2) % nv
    outs = ctx.sssp_batch([(G, src), (G, other)], variant=variant, max_iteration=100000)[0]
    assert np.array_equal(outs[0], want) and np.array_equal(outs[1], oracle.sssp(off, idx, w, other))
    G.close()


@pytest.mark.parametrize("algo", ["sssp", "bc"])
@pytest.mark.parametrize("variant", ["async_pull_dd", "auto"])
def test_batch_teams_take_graphs_in_turn(ctx, algo, variant):
    """Far more queries than teams, over graphs whose tiles hold different rows: a team's tile rows are
    rewritten for each query it claims."""
    graphs, wants = [], []
    for k, (nv, m) in enumerate([(3000, 40000), (40, 9000), (20000, 41000), (700, 20001)]):
        s, d = _random(nv, m, 17 * k + nv)
        if algo == "sssp":
            off, idx, w = _csr(nv, s, d, np.random.default_rng(k).integers(1, 1000, m).astype(np.uint32))
            graphs.append(ctx.graph_from_csr(off, idx, w))
            wants.append([oracle.sssp(off, idx, w, src) for src in range(3)])
        else:
            off, idx, _ = _csr(nv, s, d)
            graphs.append(ctx.graph_from_csr(off, idx))
            wants.append([oracle.bc_f64(off, idx, src)[0] for src in range(3)])
    picks = [(q % 4, (q // 4) % 3) for q in range(600)]
    call = ctx.sssp_batch if algo == "sssp" else ctx.bc_batch
    outs = call([(graphs[g], src) for g, src in picks], team_blocks=4, blocks_per_sm=1, variant=variant,
                max_iteration=100000)[0]
    for (g, src), out in zip(picks, outs):
        if algo == "sssp":
            assert np.array_equal(out, wants[g][src])
        else:
            assert np.all(np.abs(out - wants[g][src]) <= 1e-4 * np.abs(wants[g][src]) + 1e-5)
    for G in graphs:
        G.close()


@pytest.mark.parametrize("nv,m", TILES + [(20000, 320000)])
@pytest.mark.parametrize("variant", ["sync_pull_td", "async_push_dd", "auto"])
@pytest.mark.parametrize("no_csc", [False, True])
def test_pagerank_tiles_and_dense_push(ctx, nv, m, variant, no_csc):
    if no_csc and variant != "async_push_dd":
        pytest.skip("pull needs the in-edge view")
    s, d = _random(nv, m, nv * 3 + m)
    off, idx, _ = _csr(nv, s, d)
    want = oracle.pagerank_fixed_point_f64(off, idx)[0]
    G = ctx.graph_from_csr(off, idx, no_csc=no_csc)
    r = G.pagerank(variant=variant, pr_error=1e-8, max_iteration=100000)[0].astype(np.float64)
    assert np.abs(r / r.sum() - want / want.sum()).sum() <= 1e-6
    G.close()


@pytest.mark.parametrize("variant", ["auto", "async_push_dd", "async_pull_dd"])
def test_batches_by_density(ctx, variant):
    """Batches of sparse graphs alone, of dense ones alone and of both take different kernels."""
    graphs = []
    for nv, s, d in (_cliques(40, 12), _cliques(3000, 3)):
        off, idx, _ = _csr(nv, s, d)
        graphs.append((ctx.graph_from_csr(off, idx, symmetric=True), off, idx))
    kw = dict(variant=variant, max_iteration=100000)
    for picks in ([0], [1], [0, 1]):
        queries = [(graphs[g][0], src) for g in picks for src in (0, 7, 450)]
        levels = ctx.bfs_batch(queries, **kw)[0]
        deps = ctx.bc_batch(queries, **kw)[0]
        for (g, src), lv, dep in zip([(g, src) for g in picks for src in (0, 7, 450)], levels, deps):
            _, off, idx = graphs[g]
            assert np.array_equal(lv, oracle.bfs(off, idx, src))
            want = oracle.bc_f64(off, idx, src)[0]
            assert np.all(np.abs(dep - want) <= 1e-4 * np.abs(want) + 1e-5)
    for G, _, _ in graphs:
        G.close()


@pytest.mark.parametrize("variant", ["auto", "async_push_dd"])
def test_bc_above_the_dense_size(ctx, variant):
    h = sg.HostGraph.rmat(21, 16, symmetric=True, seed=1)
    G = ctx.graph(h, symmetric=True)
    src = int(h.pick_sources(1, 3)[0])
    bc, sigma, _ = G.bc(src, variant=variant)
    want, sig, _ = oracle.bc_f64(h.offsets, h.indices, src)
    assert np.array_equal(sigma.astype(np.float64), sig)
    assert np.all(np.abs(bc - want) <= 1e-4 * np.abs(want) + 1e-5)
    G.close()


def test_default_sssp_batch_without_in_edges(ctx):
    """A graph without in-edges makes the whole batch push, hub chunks included."""
    queries, wants = [], []
    for k, no_csc in ((700, True), (2000, False)):
        nv, s, d = _hub(k)
        off, idx, w = _csr(nv, np.concatenate([s, d]), np.concatenate([d, s]),
                           np.random.default_rng(k).integers(1, 64, 2 * len(s)).astype(np.uint32))
        G = ctx.graph_from_csr(off, idx, w, no_csc=no_csc)
        for src in (0, nv - 1, 5):
            queries.append((G, src))
            wants.append(oracle.sssp(off, idx, w, src))
    outs = ctx.sssp_batch(queries, max_iteration=100000)[0]
    assert all(np.array_equal(x, y) for x, y in zip(outs, wants))
    for G in {id(g): g for g, _ in queries}.values():
        G.close()


def _near_far_rounds(nv, off, idx, w, src, delta):
    """(in_nodes, out_nodes, in_workload, out_workload) of every near/far round on a tree, where each vertex gets its
    distance once and the rounds do not depend on the order of the work."""
    deg = np.diff(off.astype(np.int64))
    dist = {src: 0}
    near, far, limit, rounds, pile = [src], set(), delta, [], False
    work = lambda vs: int(sum(deg[v] for v in vs))
    while near or far:
        if pile:
            take = [v for v in far if dist[v] < limit]
            n_in, w_in = len(far), work(far)
            far -= set(take)
        else:
            take, n_in, w_in = near, len(near), work(near)
        near = []
        for u in take:
            for e in range(off[u], off[u + 1]):
                v = int(idx[e])
                dist[v] = dist[u] + int(w[e])
                if dist[v] < limit:
                    near.append(v)
                else:
                    far.add(v)
        rounds.append((n_in, len(near) + len(far), w_in, work(near) + work(far)))
        pile = not near
        if pile:
            limit += delta
    return rounds


@pytest.mark.parametrize("lb", ["fine", "none"])
@pytest.mark.parametrize("fan,nv", [(3, 4000), (12, 9000)])
def test_trace_of_near_far_rounds(ctx, lb, fan, nv):
    child = np.arange(1, nv, dtype=np.uint32)
    off, idx, w = _csr(nv, (child - 1) // fan, child, np.random.default_rng(fan).integers(1, 50, nv - 1).astype(np.uint32))
    G = ctx.graph_from_csr(off, idx, w)
    dist, st, tr = G.sssp(0, variant="async_push_dd", priority="low_high", priority_delta=20, lb_push=lb,
                          max_iteration=100000, trace_capacity=4096)
    assert np.array_equal(dist, oracle.sssp(off, idx, w, 0))
    want = _near_far_rounds(nv, off, idx, w, 0, 20)
    got = [(t["in_nodes"], t["out_nodes"], t["in_workload"], t["out_workload"]) for t in tr]
    assert got == want
    G.close()


def test_trace_of_topology_driven_bc_pull(ctx):
    """out_nodes of a topology-driven round = the vertices that are active after it: those with a level so far (and in
    the first round the source once more, active at the start)."""
    nv, s, d = _hub(700)
    off, idx, _ = _csr(nv, s, d)
    level = oracle.bfs(off, idx, 0)
    G = ctx.graph_from_csr(off, idx)
    bc, sigma, st = G.bc(0, variant="sync_pull_td", max_iteration=6, trace_capacity=64)
    assert st.n_trace == 6
    assert [st.trace[r].out_nodes for r in range(6)] == [int((level <= r + 1).sum()) + (r == 0) for r in range(6)]
    G.close()


def _gap(nv, m, at, gap, seed):
    """A random graph whose ids from `at` on are moved up by `gap` unused ones."""
    s, d = _random(nv, m, seed)
    up = lambda x: np.where(x >= at, x + gap, x).astype(np.uint32)
    return nv + gap, up(s), up(d)


# gaps around the rows a tile ranks (1024) and the rows an entry tile walks (65536), at the start, inside and at the end
@pytest.mark.parametrize("gap", [1000, 1030, 65500, 70000])
@pytest.mark.parametrize("at", [0, 1500, 3000])
def test_runs_of_unused_ids(ctx, gap, at):
    nv, s, d = _gap(3000, 40000, at, gap, gap + at)
    w = np.random.default_rng(gap).integers(1, 1000, len(s)).astype(np.uint32)
    src = int(s[0])
    off, idx, ww = _csr(nv, s, d, w)
    G = ctx.graph_from_csr(off, idx, ww)
    for variant in ("async_pull_dd", "sync_pull_td", "auto"):
        assert np.array_equal(G.sssp(src, variant=variant, max_iteration=100000)[0], oracle.sssp(off, idx, ww, src))
    bc, sigma, _ = G.bc(src, variant="async_pull_dd")
    want, sig, _ = oracle.bc_f64(off, idx, src)
    assert np.array_equal(sigma.astype(np.float64), sig)
    assert np.all(np.abs(bc - want) <= 1e-4 * np.abs(want) + 1e-5)
    want = oracle.pagerank_fixed_point_f64(off, idx)[0]
    for variant in ("sync_pull_td", "async_push_dd"):
        r = G.pagerank(variant=variant, pr_error=1e-8, max_iteration=100000, lb_push="fine")[0].astype(np.float64)
        assert np.abs(r / r.sum() - want / want.sum()).sum() <= 1e-6
    coff, cidx, cw = G.copy_out(csc=True)
    G.close()
    tc = oracle.csr_tocsc(off, idx, ww)
    assert np.array_equal(coff, tc[0]) and np.array_equal(cidx, tc[1]) and np.array_equal(cw, tc[2])


def test_unused_ids_cost_their_passes_only(ctx):
    """10 pull rounds with 4 M unused ids between two halves of a graph: a few passes over the ids (about 0.2 ms a
    round), where a warp that steps through them 32 at a time takes over 60 ms a round."""
    ms = []
    for gap in (0, 1 << 22):
        nv, s, d = _gap(65536, 1 << 20, 32768, gap, 5)
        off, idx, _ = _csr(nv, s, d)
        G = ctx.graph_from_csr(off, idx)
        ms.append(min(G.pagerank(variant="sync_pull_td", max_iteration=10)[1].time_kernel_ms for _ in range(3)))
        G.close()
    assert ms[1] < ms[0] + 50, ms


# entries around one radix tile (4096), ids around a digit (8 bits) and several
BUILDS = [(1, 5), (2, 4095), (255, 4096), (256, 4097), (257, 8192), (65536, 8193), (65537, 20000), (70000, 3)]


@pytest.mark.parametrize("nv,m", BUILDS)
@pytest.mark.parametrize("code", range(8))
@pytest.mark.parametrize("sort_rows", [False, True])
def test_build_radix_edges(ctx, nv, m, code, sort_rows):
    s, d = _random(nv, m, nv + 7 * m)
    if nv > 10:
        s[: m // 3] = 3  # one long row
    w = np.random.default_rng(m).integers(0, 2**32, m, dtype=np.uint64).astype(np.uint32)
    want = oracle.gtools_build(nv, s, d, w, deself_cycle=bool(code & 1), deduplicate=bool(code & 2), d2ud=bool(code & 4),
                               sort_rows=sort_rows)
    G = ctx.build_graph(nv, s, d, w, deself_cycle=bool(code & 1), deduplicate=bool(code & 2), d2ud=bool(code & 4),
                        sort_rows=sort_rows)
    off, idx, ww = G.copy_out()
    coff, cidx, cw = G.copy_out(csc=True)
    G.close()
    assert all(np.array_equal(x, y) for x, y in zip((off, idx, ww), want))
    tc = oracle.csr_tocsc(off, idx, ww)
    assert np.array_equal(coff, tc[0]) and np.array_equal(cidx, tc[1]) and np.array_equal(cw, tc[2])


def _cliques(n, k):
    """A path of n cliques of k vertices: average degree about k - 1, about n levels."""
    s, d = [], []
    for c in range(n):
        v = np.arange(c * k, (c + 1) * k, dtype=np.uint32)
        a, b = np.meshgrid(v, v)
        keep = a != b
        s.append(a[keep]), d.append(b[keep])
        if c:
            s.append(np.array([c * k - 1, c * k], np.uint32)), d.append(np.array([c * k, c * k - 1], np.uint32))
    return n * k, np.concatenate(s), np.concatenate(d)


@pytest.mark.parametrize("n", [4, 8, 15, 30])  # up to 59 levels: below, at and past the 16 levels of the planes
@pytest.mark.parametrize("nsrc", [1, 33, 64])
@pytest.mark.parametrize("variant", ["auto", "async_push_dd", "async_pull_dd"])
def test_msbfs_levels_past_planes(ctx, n, nsrc, variant):
    nv, s, d = _cliques(n, 12)
    off, idx, _ = _csr(nv, s, d)
    src = np.random.default_rng(n).integers(0, nv, nsrc).astype(np.uint32)
    src[0] = 0
    G = ctx.graph_from_csr(off, idx, symmetric=True)
    rows, st = G.msbfs(src, variant=variant)
    want = np.stack([oracle.bfs(off, idx, int(x)) for x in src])
    assert np.array_equal(rows, want)
    for limit in (1, 3, 14, 15, 16, 17, 40):
        rows, _ = G.msbfs(src, variant=variant, max_iteration=limit)
        assert np.array_equal(rows, np.where(want <= limit, want, np.uint32(0xFFFFFFFF))), limit
    G.close()


@pytest.mark.parametrize("nv,m", [(1, 0), (3, 2), (700, 9000), (5000, 60000)])
def test_reached_counts(ctx, nv, m):
    s, d = _random(nv, m, nv + m)
    off, idx, _ = _csr(nv, s, d)
    deg = np.diff(off.astype(np.int64))
    G = ctx.graph_from_csr(off, idx)
    for call in (G.bfs, G.sssp):
        val, st, _ = call(0)
        reached = val != 0xFFFFFFFF
        assert st.vertices_reached == reached.sum() and st.edges_reached == deg[reached].sum()
        assert st.search_depth == val[reached].max()
    G.close()
