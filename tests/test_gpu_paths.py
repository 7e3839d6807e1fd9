"""Traversal paths at the sizes where their dispatch changes: results against
the CPU oracle (integers bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stars(gsrb, degrees, seed=1, whi=255):
    """Hubs of the given degrees on a common pool of leaves, joined in a path."""
    rng = np.random.default_rng(seed)
    pool = max(degrees) + 16
    src, dst = [], []
    for i, d in enumerate(degrees):
        leaves = rng.choice(pool, d - 1 - (0 < i < len(degrees) - 1), replace=False)  # path edges count too
        src.append(np.full(leaves.size, pool + i))
        dst.append(leaves)
    k = len(degrees)
    src.append(pool + np.arange(k - 1))
    dst.append(pool + np.arange(1, k))
    return gsrb.csr_from_edges(pool + k, np.concatenate(src), np.concatenate(dst), whi=whi), pool


@pytest.fixture(scope="module")
def path_graphs(gsrb):
    rng = np.random.default_rng(3)
    left, right = 2600, 300  # 2600 vertices of degree > 256: more hubs than one shared-memory list holds
    bip = gsrb.csr_from_edges(left + right, np.repeat(np.arange(left), 260),
                              left + np.concatenate([rng.choice(right, 260, replace=False) for _ in range(left)]))
    return {
        "degrees": _stars(gsrb, [255, 256, 257, 258, 31, 32, 33, 4095, 4096, 4097, 2])[0],
        "bipartite": bip,
        "grid": gsrb.grid2d(301, 77, seed=9),
        "rmat": gsrb.rmat(13, 20, seed=5),
    }


@pytest.mark.parametrize("name", ["degrees", "bipartite", "grid", "rmat"])
@pytest.mark.parametrize("shape", ["default", "one_cta", "three_ctas"])
@pytest.mark.parametrize("delta", [3, 700, 1 << 30])
def test_sssp_paths(gsrb, ctx, orc, path_graphs, name, shape, delta):
    g = path_graphs[name]
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.int32)
    c = None if shape == "default" else gsrb.cfg(variant=gsrb.BAR_FANOUT, threads=96,
                                                 grid_override=1 if shape == "one_cta" else 3)
    for src in (0, g.nnodes - 1):
        rc, _ = dg.sssp(src, out, delta, c)
        gsrb.check(rc, "sssp")
        assert np.array_equal(out.download(), orc.dijkstra(g, src))


def test_sssp_long_weights(gsrb, ctx, orc):
    """Path lengths beyond INT_MAX are no paths (the sum saturates)."""
    n = 12
    g = gsrb.csr_from_edges(n, np.arange(n - 1), np.arange(1, n))
    w = np.where(g.edge_data > 0, 2**29, 0).astype(np.int32)
    g = gsrb.Graph(g.row_start, g.edge_dst, w)
    dg = ctx.graph(g)
    out = ctx.array(n, np.int32)
    rc, _ = dg.sssp(0, out, 1 << 30)
    gsrb.check(rc, "sssp")
    want = [min(i * 2**29, 2**31 - 1) for i in range(4)] + [2**31 - 1] * (n - 4)
    assert out.download().tolist() == want


def test_batch_calls_back_to_back(gsrb, ctx, orc, path_graphs):
    """Calls on one batch without a wait between them, each with other sources:
    the last call's results stand."""
    gs = [path_graphs["grid"], path_graphs["degrees"], path_graphs["rmat"]]
    dgs = [ctx.graph(g) for g in gs]
    outs = [[ctx.array(g.nnodes, np.int32) for g in gs] for _ in range(6)]
    b = gsrb.Batch(ctx, dgs)
    for i in range(6):
        gsrb.check(b.sssp([i] * 3, outs[i], 500) if i % 2 else b.bfs([i] * 3, outs[i]), "batch")
    rc, _ = b.stats()
    gsrb.check(rc)
    for i in range(6):
        for g, o in zip(gs, outs[i]):
            assert np.array_equal(o.download(), orc.dijkstra(g, i) if i % 2 else orc.bfs(g, i))


def _thin_graphs(gsrb):
    rng = np.random.default_rng(11)
    n = 6000
    # a chain of fans: levels of 1, then many, then 1 vertices (cluster -> grid -> cluster)
    fans, src, dst, base = [40, 700, 30000, 3, 20000, 1], [], [], 0
    for f in fans:
        src.append(np.full(f, base))
        dst.append(base + 1 + np.arange(f))
        src.append(base + 1 + np.arange(f))
        dst.append(np.full(f, base + f + 1))
        base += f + 1
    fan = gsrb.csr_from_edges(base + 1, np.concatenate(src), np.concatenate(dst))
    # random tree plus chords: degrees 1 to about 12, long
    par = np.maximum(0, np.arange(1, n) - 1 - rng.integers(0, 6, n - 1))
    tree = gsrb.csr_from_edges(n, np.concatenate([par, rng.integers(0, n, 40)]),
                               np.concatenate([np.arange(1, n), rng.integers(0, n, 40)]))
    return {
        "fans": fan,
        "tree": tree,
        "wide": gsrb.grid2d(3000, 40, seed=2),
        "square": gsrb.grid2d(600, 600, seed=4),
        "path": gsrb.csr_from_edges(5000, np.arange(4999), np.arange(1, 5000)),
        "isolated": gsrb.csr_from_edges(70, [0, 1, 50], [1, 2, 51]),
        "rmat": gsrb.rmat(15, 12, seed=8),
        "directed": gsrb.csr_from_edges(4000, np.arange(3999), np.arange(1, 4000), symmetrize=False),
    }


@pytest.fixture(scope="module")
def thin_graphs(gsrb):
    return _thin_graphs(gsrb)


@pytest.mark.parametrize("name", ["fans", "tree", "wide", "square", "path", "isolated", "rmat", "directed"])
@pytest.mark.parametrize("variant", [None, 6, 8, 9])
def test_bfs_thin_levels(gsrb, ctx, orc, thin_graphs, name, variant):
    """Levels that run on one cluster, and the hand-overs between it and the grid."""
    g = thin_graphs[name]
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.int32)
    c = None if variant is None else gsrb.cfg(variant=variant, ctas_per_sm=1, threads=256)
    for src in (0, g.nnodes // 2, g.nnodes - 1):
        rc, st = dg.bfs(src, out, gsrb.BFS_HEURISTIC, c)
        gsrb.check(rc, "bfs")
        ctx.check_status("bfs")
        want = orc.bfs(g, src)
        assert np.array_equal(out.download(), want)
        assert st.edges == orc.traversed_edges(g, want)
        assert st.levels == int(want[want != 2**31 - 1].max()) + 1 if want.max() >= 0 else 0
        tr = dg.trace()
        assert tr["level"].tolist() == list(range(1, len(tr) + 1))
        assert int(tr["nf"].sum()) == int((want != 2**31 - 1).sum())


@pytest.mark.parametrize("name", ["fans", "tree", "wide", "square", "path", "isolated", "directed"])
@pytest.mark.parametrize("delta", [40, 1000, 1 << 30])
def test_sssp_thin_graphs(gsrb, ctx, orc, thin_graphs, name, delta):
    """Thin graphs: rounds on one cluster, and the hand-over of the rest to the
    grid (the fans outgrow the cluster's queues, the wide buckets its far piles)."""
    g = thin_graphs[name]
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.int32)
    for src in (0, g.nnodes // 2):
        rc, st = dg.sssp(src, out, delta)
        gsrb.check(rc, "sssp")
        ctx.check_status("sssp")
        want = orc.dijkstra(g, src)
        assert np.array_equal(out.download(), want)
        assert st.levels >= 1 and st.edges >= orc.traversed_edges(g, want) and st.delta == delta


@pytest.mark.parametrize("name", ["degrees", "bipartite", "grid", "rmat", "tree", "isolated", "path"])
@pytest.mark.parametrize("shape", ["default", "one_cta"])
def test_pagerank_residual_rounds(gsrb, ctx, orc, path_graphs, thin_graphs, name, shape):
    """Pulled and pushed rounds of the residual PageRank against the FP64 fixed
    point: what is left over is below epsilon a vertex, which the chain of
    pushes amplifies by at most 1 / (1 - alpha); FP32 sums add 1e-6."""
    g = path_graphs.get(name) or thin_graphs[name]
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.float32)
    c = None if shape == "default" else gsrb.cfg(variant=gsrb.BAR_FANOUT, threads=128, grid_override=1)
    ref = orc.pagerank_push(g, 0.85, 200)
    for eps in (1e-6, 1e-3):
        rc, st = dg.pagerank_residual(out, 0.85, eps, c=c)
        gsrb.check(rc, "pagerank_residual")
        ctx.check_status("pagerank_residual")
        assert st.levels >= 1
        assert np.abs(out.download() - ref).sum() <= (eps / 0.15 + 2e-6) * g.nnodes + 2e-6 * ref.sum()
    rc, st = dg.pagerank_residual(out, 0.85, 1e-9, 3, c)
    gsrb.check(rc, "pagerank_residual")
    assert st.levels == 3 or name == "isolated"


@pytest.mark.parametrize("name", ["degrees", "bipartite", "grid", "rmat"])
@pytest.mark.parametrize("mode", [1, 3])  # heuristic, pull every level after the first
def test_bfs_pull_rows(gsrb, ctx, orc, path_graphs, name, mode):
    """Pull levels over rows at the edges of the lane / warp split (4, 32, 128 edges)."""
    g = path_graphs[name]
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.int32)
    for src in (0, 7, g.nnodes - 1):
        for c in (None, gsrb.cfg(variant=gsrb.BAR_FANOUT, threads=64, grid_override=3)):
            rc, st = dg.bfs(src, out, mode, c)
            gsrb.check(rc, "bfs")
            want = orc.bfs(g, src)
            assert np.array_equal(out.download(), want)
            assert st.edges == orc.traversed_edges(g, want)


@pytest.mark.parametrize("tail", [1, 700])
def test_sssp_vertices_without_out_edges(gsrb, ctx, orc, tail):
    """Directed rows that end at the arrays' end: nothing is read for them."""
    n = 1500
    src = np.concatenate([np.arange(n - 1), np.arange(tail) % n])
    dst = np.concatenate([np.arange(1, n), n + np.arange(tail)])
    g = gsrb.csr_from_edges(n + tail, src, dst, symmetrize=False)
    dg = ctx.graph(g)
    out = ctx.array(g.nnodes, np.int32)
    for source in (0, n + tail - 1):
        for delta in (50, 1 << 30):
            rc, st = dg.sssp(source, out, delta)
            gsrb.check(rc, "sssp")
            assert np.array_equal(out.download(), orc.dijkstra(g, source))
        rc, st = dg.bfs(source, out)
        gsrb.check(rc, "bfs")
        assert np.array_equal(out.download(), orc.bfs(g, source))


@pytest.mark.parametrize("name", ["path", "wide", "tree"])
def test_explicit_launch_runs_alone(gsrb, ctx, orc, thin_graphs, name):
    """A launch configuration of the caller's runs the whole traversal: one
    launch, whatever the graph; without one thin steps run on the cluster."""
    g = thin_graphs[name]
    dg = ctx.graph(g)
    dg.set_policy(gsrb.mlp_init(77))
    out = ctx.array(g.nnodes, np.int32)

    def launches(call):
        n0 = gsrb.launch_count()
        rc, st = call()
        gsrb.check(rc, "traversal")
        return gsrb.launch_count() - n0

    want, dist = orc.bfs(g, 0), orc.dijkstra(g, 0)
    for variant in (gsrb.BAR_SOFT2, gsrb.BAR_FLAT, gsrb.BAR_CCG, gsrb.BAR_FANOUT):
        c = gsrb.cfg(variant=variant, ctas_per_sm=1, threads=128, cluster=1)
        for mode in (gsrb.BFS_HEURISTIC, gsrb.BFS_LEARNED):
            assert launches(lambda: dg.bfs(0, out, mode, c)) == 1
            assert np.array_equal(out.download(), want)
        assert launches(lambda: dg.sssp(0, out, 400, c)) == 1
        assert 3 not in dg.trace()["dir"]
        assert np.array_equal(out.download(), dist)
    assert launches(lambda: dg.bfs(0, out)) >= 2 and launches(lambda: dg.sssp(0, out, 400)) >= 2
    assert np.all(dg.trace()["dir"] == 3)


def test_batch_replay_between_live_calls(gsrb, ctx, orc, path_graphs):
    """A replay runs the captured call, whatever ran live before the capture,
    between it and the replay, or is enqueued right behind the replay."""
    gs = [path_graphs["grid"], path_graphs["degrees"]]
    dgs = [ctx.graph(g) for g in gs]
    b = gsrb.Batch(ctx, dgs)
    outs = {k: [ctx.array(g.nnodes, np.int32) for g in gs] for k in ("live", "bfs", "sssp")}

    def live(src):
        gsrb.check(b.bfs([src] * 2, outs["live"], gsrb.BFS_PUSH), "live")

    def holds(key, f):
        for g, o in zip(gs, outs[key]):
            assert np.array_equal(o.download(), f(g))

    live(3)
    execs = []
    for key in ("bfs", "sssp"):  # two captured calls on one batch
        cg = gsrb.CudaGraph(ctx)
        with cg:
            gsrb.check(b.bfs([7] * 2, outs[key]) if key == "bfs" else b.sssp([9] * 2, outs[key], 500), "captured")
        execs.append(cg)
    live(11)
    for _ in range(3):
        for key in ("bfs", "sssp"):
            for o in outs[key]:
                o.zero()
        live(5)
        execs[0].launch()
        live(12)
        execs[1].launch()
        live(13)
        gsrb.check(b.stats()[0], "stats")
        holds("bfs", lambda g: orc.bfs(g, 7))
        holds("sssp", lambda g: orc.dijkstra(g, 9))
        holds("live", lambda g: orc.bfs(g, 13))
    for cg in execs:
        cg.free()
    b.free()


def test_batch_first_call_captured(gsrb, ctx, orc, path_graphs):
    """The first call on a batch, of a shape not launched before, may be a captured one."""
    gs = [path_graphs["grid"], path_graphs["rmat"]]
    outs = [ctx.array(g.nnodes, np.int32) for g in gs]
    b = gsrb.Batch(ctx, [ctx.graph(g) for g in gs], gsrb.cfg(variant=gsrb.BAR_FLIP, ctas_per_sm=1, threads=352))
    cg = gsrb.CudaGraph(ctx)
    with cg:
        gsrb.check(b.sssp([4] * 2, outs, 700), "captured")
    cg.launch()
    gsrb.check(b.stats()[0], "stats")
    for g, o in zip(gs, outs):
        assert np.array_equal(o.download(), orc.dijkstra(g, 4))
    cg.free()
    b.free()
