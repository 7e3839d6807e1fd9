"""A graph used from another context than the one it was made on: the calling
context runs the traversal and reports its status."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def two(gsrb, ctx):
    """(graph, device graph made on a second context, then used from the first)"""
    graphs = {"rmat": gsrb.rmat(12, 16, seed=21), "grid": gsrb.grid2d(90, 70, seed=22)}
    maker = gsrb.Context(0)
    dgs = {}
    for k, g in graphs.items():
        dgs[k] = maker.graph(g)
        dgs[k].ctx = ctx
    yield graphs, dgs
    for dg in dgs.values():
        dg.free()
    maker.close()


@pytest.mark.parametrize("name", ["rmat", "grid"])
def test_traversals_from_another_context(gsrb, ctx, orc, two, name):
    graphs, dgs = two
    g, dg = graphs[name], dgs[name]
    out, rank = ctx.array(g.nnodes, np.int32), ctx.array(g.nnodes, np.float32)
    for src in (0, 17, g.nnodes - 1):
        want = orc.bfs(g, src)
        for mode in (gsrb.BFS_HEURISTIC, gsrb.BFS_PUSH):
            rc, st = dg.bfs(src, out, mode)
            gsrb.check(rc, "bfs")
            assert np.array_equal(out.download(), want)
            assert st.edges == orc.traversed_edges(g, want) and st.levels == want[want != 2**31 - 1].max() + 1
            assert 0 < st.kernel_ms < 1e4
        rc, st = dg.sssp(src, out, 300)
        gsrb.check(rc, "sssp")
        assert np.array_equal(out.download(), orc.dijkstra(g, src))
        assert st.delta == 300 and st.levels >= 1
    rc, st = dg.pagerank(rank, 0.85, 20)
    gsrb.check(rc, "pagerank")
    assert st.levels == 20 and orc.normalized_l1(rank.download(), orc.pagerank(g, 0.85, 20)) <= 1e-6
    rc, st = dg.pagerank_residual(rank, 0.85, 1e-6)
    gsrb.check(rc, "pagerank_residual")
    assert st.levels >= 1


def test_batch_from_another_context(gsrb, ctx, orc, two):
    graphs, dgs = two
    names = list(graphs)
    outs = [ctx.array(graphs[k].nnodes, np.int32) for k in names]
    b = gsrb.Batch(ctx, [dgs[k] for k in names])
    for src in (3, 40):
        gsrb.check(b.bfs([src] * 2, outs), "batch")
        rc, st = b.stats()
        gsrb.check(rc, "stats")
        for k, o, s in zip(names, outs, st):
            want = orc.bfs(graphs[k], src)
            assert np.array_equal(o.download(), want)
            assert s.edges == orc.traversed_edges(graphs[k], want)
    b.free()
