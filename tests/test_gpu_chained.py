"""Chained reductions (cfg.overlap) read a finished input whatever ran before
their predecessor on the stream: the predecessor alone may not write it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1 << 22  # one CTA sums it for a while; the small launches behind it fit beside it


def _cfg(gsrb, **kw):
    return gsrb.cfg(variant=gsrb.BAR_FANOUT, threads=256, grid_override=1, tile=1, **kw)


@pytest.fixture(scope="module")
def arrays(gsrb, ctx):
    a = np.full(N, 3, np.int32)
    return {"big": ctx.to_device(a), "small": ctx.to_device(np.arange(1000, dtype=np.int32)),
            "res": ctx.array(4, np.int64), "want": 3 * N}


@pytest.mark.parametrize("replayed", [False, True])
def test_behind_a_plain_reduction(gsrb, ctx, arrays, replayed):
    """plain reduce -> chained reduce of another array -> chained reduce of the
    plain one's result (two int32 words, the upper zero)."""
    d, plain, chained = arrays, _cfg(gsrb), _cfg(gsrb, overlap=1)

    def calls():
        gsrb.check(ctx.reduce_i32(d["big"], N, d["res"].at(0), plain), "plain")
        gsrb.check(ctx.reduce_i32(d["small"], 1000, d["res"].at(1), chained), "chained")
        gsrb.check(ctx.reduce_i32(d["res"].at(0), 2, d["res"].at(2), chained), "chained")

    g = None
    if replayed:
        g = gsrb.CudaGraph(ctx)
        with g:
            calls()
    for _ in range(4):
        d["res"].zero()
        g.launch() if g else calls()
        ctx.check_status("chain")
        assert d["res"].download().tolist() == [d["want"], 499500, d["want"], 0]
    if g:
        g.free()


def test_behind_a_replay(gsrb, ctx, arrays):
    """A replayed graph may end in a kernel that lets the next one in early."""
    d, plain, chained = arrays, _cfg(gsrb), _cfg(gsrb, overlap=1)
    g = gsrb.CudaGraph(ctx)
    with g:
        gsrb.check(ctx.reduce_i32(d["big"], N, d["res"].at(0), plain), "plain")
    for _ in range(4):
        d["res"].zero()
        g.launch()
        gsrb.check(ctx.reduce_i32(d["small"], 1000, d["res"].at(1), chained), "chained")
        gsrb.check(ctx.reduce_i32(d["res"].at(0), 2, d["res"].at(2), chained), "chained")
        ctx.check_status("chain")
        assert d["res"].download().tolist() == [d["want"], 499500, d["want"], 0]
    g.free()


def test_behind_chained_reductions(gsrb, ctx, arrays):
    """Every third call reads the result of the chained call before the one
    before it; more results than the context keeps in mind."""
    d, chained = arrays, _cfg(gsrb, overlap=1)
    k = 100
    res = ctx.array(3 * k, np.int64).zero()
    for i in range(k):
        gsrb.check(ctx.reduce_i32(d["big"], N, res.at(3 * i), chained), "chained")
        gsrb.check(ctx.reduce_i32(d["small"], 1000, res.at(3 * i + 1), chained), "chained")
        gsrb.check(ctx.reduce_i32(res.at(3 * i), 2, res.at(3 * i + 2), chained), "chained")
    ctx.check_status("chain")
    assert res.download().tolist() == [d["want"], 499500, d["want"]] * k
    res.zero()
    for i in range(k):  # as many results without a reader: the chain starts over when the list is full
        gsrb.check(ctx.reduce_i32(d["small"], 1000, res.at(i), chained), "chained")
    gsrb.check(ctx.reduce_i32(res, 2 * k, res.at(k), chained), "chained")
    ctx.check_status("chain")
    assert res.download().tolist()[:k + 1] == [499500] * k + [499500 * k]
