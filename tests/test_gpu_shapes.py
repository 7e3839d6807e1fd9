"""Launch shapes of many small CTAs: traversals accept every shape their CTAs fit
without the append stages, and give the same results with and without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shape_graphs(gsrb):
    rng = np.random.default_rng(5)
    hub = np.concatenate([np.zeros(20000, np.int64), rng.integers(1, 20001, 60000)])
    return {"rmat": gsrb.rmat(14, 16, seed=31), "grid": gsrb.grid2d(120, 90, seed=32),
            # a hub of more than 4096 edges ahead of pull levels
            "hub": gsrb.csr_from_edges(20001, hub, np.concatenate([np.arange(1, 20001), rng.integers(1, 20001, 60000)]))}


@pytest.mark.parametrize("name", ["rmat", "grid", "hub"])
@pytest.mark.parametrize("per_sm,threads", [(8, 128), (7, 128), (8, 64), (5, 128), (4, 128), (2, 512)])
def test_traversal_shapes(gsrb, ctx, orc, shape_graphs, name, per_sm, threads):
    g = shape_graphs[name]
    dg = ctx.graph(g)
    c = gsrb.cfg(variant=gsrb.BAR_FANOUT, ctas_per_sm=per_sm, threads=threads)
    out, rank = ctx.array(g.nnodes, np.int32), ctx.array(g.nnodes, np.float32)
    dist, level = orc.dijkstra(g, 0), orc.bfs(g, 0)
    for delta in (100, 10000):
        gsrb.check(dg.sssp(0, out, delta, c)[0], "sssp")
        assert np.array_equal(out.download(), dist)
    gsrb.check(dg.pagerank_residual(rank, 0.85, 1e-6, c=c)[0], "pagerank_residual")
    ref = orc.pagerank_push(g, 0.85, 200)
    # what is left over is below epsilon a vertex, amplified by at most 1 / (1 - alpha); FP32 sums add 2e-6
    assert np.abs(rank.download() - ref).sum() <= (1e-6 / 0.15 + 2e-6) * g.nnodes + 2e-6 * ref.sum()
    b = gsrb.Batch(ctx, [dg], c)
    gsrb.check(b.sssp([0], [out], 300), "batch sssp")
    gsrb.check(b.stats()[0], "batch sssp")
    assert np.array_equal(out.download(), dist)
    # BFS keeps the policy's weights and the hub lists: seven CTAs, six with a batch's descriptor
    c.ctas_per_sm = min(per_sm, 6)
    b = gsrb.Batch(ctx, [dg], c)
    c.ctas_per_sm = min(per_sm, 7)
    for mode in (gsrb.BFS_HEURISTIC, gsrb.BFS_PUSH, gsrb.BFS_TOPO):
        gsrb.check(dg.bfs(0, out, mode, c)[0], "bfs")
        assert np.array_equal(out.download(), level)
        gsrb.check(b.bfs([0], [out], mode), "batch bfs")
        gsrb.check(b.stats()[0], "batch bfs")
        assert np.array_equal(out.download(), level)
