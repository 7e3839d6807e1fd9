"""A traversal whose grid cannot be co-resident is refused as a whole: with its
status, and with the caller's array untouched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["cfg", "launch_choice"])
@pytest.mark.parametrize("name", ["thin", "fat"])
def test_refused_traversals_write_nothing(gsrb, ctx, orc, name, how):
    g = gsrb.grid2d(300, 200, seed=3) if name == "thin" else gsrb.rmat(13, 16, seed=3)
    dg = ctx.graph(g)
    big = gsrb.cfg(variant=gsrb.BAR_FANOUT, ctas_per_sm=3, threads=1024)
    out = ctx.array(g.nnodes, np.int32)
    mark = np.full(g.nnodes, -7, np.int32)
    dg.set_policy(gsrb.mlp_init(5))
    dg.set_sssp_policy(gsrb.mlp_init(6))
    if how == "launch_choice":
        dg.set_launch_choices(big, big)
    c = big if how == "cfg" else None
    modes = [gsrb.BFS_LEARNED] if how == "launch_choice" else [gsrb.BFS_LEARNED, gsrb.BFS_HEURISTIC, gsrb.BFS_PUSH]
    for mode in modes:
        out.upload(mark)
        assert dg.bfs(0, out, mode, c)[0] == gsrb.ERR_NOT_CORESIDENT
        assert np.array_equal(out.download(), mark)
    for delta in [gsrb.SSSP_DELTA_LEARNED] if how == "launch_choice" else [gsrb.SSSP_DELTA_LEARNED, 500]:
        out.upload(mark)
        assert dg.sssp(0, out, delta, c)[0] == gsrb.ERR_NOT_CORESIDENT
        assert np.array_equal(out.download(), mark)
    dg.set_launch_choices(None, None)
    gsrb.check(dg.bfs(0, out)[0], "bfs")
    assert np.array_equal(out.download(), orc.bfs(g, 0))
    dg.free()
