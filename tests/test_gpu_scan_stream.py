"""The default scan (streaming form) against the CPU oracle: tile edges,
remainders, alignment, in place, chains of calls and graph replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# tiles are 2048 elements up to 148 of them, 8192 above; copies are whole 16-byte units
SIZES = [1, 3, 4, 5, 2047, 2048, 2049, 6 * 2048 + 1, 148 * 2048 - 1, 148 * 2048, 148 * 2048 + 1,
         148 * 8192 * 6 + 8191, 148 * 8192 * 9 + 2]


@pytest.mark.parametrize("n", SIZES)
def test_scan_u32_default(gsrb, ctx, orc, n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 2**32, n, dtype=np.uint32)  # wraps around
    d, o = ctx.to_device(a), ctx.array(n, np.uint32)
    want = orc.scan_u32(a)
    for _ in range(2):
        gsrb.check(ctx.scan(d, o, n), "scan")
    ctx.check_status("scan")
    assert np.array_equal(o.download(), want)
    gsrb.check(ctx.scan(d, d, n), "scan in place")
    ctx.check_status("scan")
    assert np.array_equal(d.download(), want)


@pytest.mark.parametrize("n", SIZES)
def test_scan_f32_default(gsrb, ctx, orc, n):
    a = gsrb.uniform_f32(n, n)
    d, o = ctx.to_device(a), ctx.array(n, np.float32)
    gsrb.check(ctx.scan(d, o, n), "scan")
    ctx.check_status("scan")
    first = o.download()
    ref = orc.scan_f32_f64(a)
    # FP32 within a warp's 128 elements (seven roundings), FP64 between, one rounding of the result
    assert np.all(np.abs(first - ref) <= 8 * 2.0**-24 * np.maximum(ref, 2.0**-24) + 1e-30)
    gsrb.check(ctx.scan(d, o, n), "scan")
    assert np.array_equal(o.download(), first)  # the same bits every time


@pytest.mark.parametrize("ioff,ooff", [(1, 0), (0, 1), (2, 2), (4, 0), (0, 4)])
def test_scan_alignment(gsrb, ctx, orc, ioff, ooff):
    n = 30011
    a = np.arange(n + 8, dtype=np.uint32)
    d, o = ctx.to_device(a), ctx.array(n + 8, np.uint32)
    o.upload(np.full(n + 8, 7, np.uint32))
    gsrb.check(ctx.scan(d.at(ioff), o.at(ooff), n), "scan")
    ctx.check_status("scan")
    got = o.download()
    assert np.array_equal(got[ooff:ooff + n], orc.scan_u32(a[ioff:ioff + n]))
    assert np.all(got[:ooff] == 7) and np.all(got[ooff + n:] == 7)


def test_scan_chain_and_replay(gsrb, ctx, orc):
    """Each call reads what the one before wrote, of several sizes, plain and replayed."""
    sizes = [100_003, 2048 * 148 + 5, 3_000_001, 17, 800_000]
    n = max(sizes)
    a = np.random.default_rng(1).integers(0, 2**32, n, dtype=np.uint32)
    want = a.copy()
    for k in sizes:
        want[:k] = orc.scan_u32(want[:k])
    d = ctx.to_device(a)
    for k in sizes:
        gsrb.check(ctx.scan(d, d, k), "scan")
    ctx.check_status("scan chain")
    assert np.array_equal(d.download(), want)
    out = ctx.array(n, np.uint32)
    with gsrb.CudaGraph(ctx) as g:
        for k in sizes:
            gsrb.check(ctx.scan(d, d, k), "scan")
        gsrb.check(ctx.scan(d, out, n), "scan")
    d.upload(a)
    g.launch()
    ctx.check_status("replay")
    assert np.array_equal(d.download(), want) and np.array_equal(out.download(), orc.scan_u32(want))
    d.upload(a)
    g.launch()
    ctx.check_status("replay")
    assert np.array_equal(d.download(), want)
    g.free()


@pytest.mark.parametrize("n", [0, 1, 5, 4099, 2 * 148 * 4 - 1, 2 * 148 * 4 + 1, 1 << 20, 3_000_001])
@pytest.mark.parametrize("grid", [0, 1, 2])  # 0: the default call
def test_reduce_in_order(gsrb, ctx, n, grid):
    """A reduction reads what the scan before it on the stream wrote, and the
    one after it may overwrite its input."""
    c = None if grid == 0 else gsrb.cfg(variant=gsrb.BAR_FANOUT, threads=256, grid_override=grid)
    a = np.random.default_rng(n).integers(0, 3, max(n, 1)).astype(np.uint32)
    d, o = ctx.to_device(a), ctx.array(max(n, 1), np.uint32)
    sums = ctx.array(4, np.int64).zero()
    want, cur = [], a[:n].astype(np.uint64)
    for k in range(4):
        gsrb.check(ctx.scan(d, d, n), "scan")
        cur = (np.cumsum(cur) - cur) & 0xffffffff if n else cur
        gsrb.check(ctx.reduce_i32(d, n, sums.at(k), c), "reduce")
        want.append(int(cur.astype(np.uint32).view(np.int32).astype(np.int64).sum()))
    ctx.check_status("chain")
    assert sums.download().tolist() == want


def test_chained_reductions_behind_a_scan(gsrb, ctx):
    """scan -> chained reduce of another array -> chained reduce of the scan's
    output: neither reduction's predecessor writes its input, so both may be
    chained, and the second must still see the whole scan."""
    n = 1 << 24
    a = np.ones(n, np.uint32)
    d, x = ctx.to_device(a), ctx.array(n, np.uint32)
    small = ctx.to_device(np.arange(1000, dtype=np.int32))
    sums = ctx.array(2, np.int64).zero()
    c = gsrb.cfg(variant=gsrb.BAR_FANOUT, ctas_per_sm=2, threads=256, overlap=1, tile=1)
    for k in range(4):
        x.zero()
        gsrb.check(ctx.scan(d, x, n), "scan")
        gsrb.check(ctx.reduce_i32(small, 1000, sums.at(0), c), "reduce")
        gsrb.check(ctx.reduce_i32(x, n, sums.at(1), c), "reduce")
        ctx.check_status("chain")
        assert sums.download().tolist() == [499500, n * (n - 1) // 2]


@pytest.mark.parametrize("big", [1e30, np.inf])
@pytest.mark.parametrize("n", [2048, 5000, 148 * 8192 * 2 + 77])
def test_scan_f32_wide_range(gsrb, ctx, n, big):
    """A value that swallows (or makes infinite) every sum behind it leaves the
    prefixes before it as they are."""
    for at in (0, n // 2, n // 2 + 77, n - 2):
        a = np.ones(n, np.float32)
        a[at] = big
        d, o = ctx.to_device(a), ctx.array(n, np.float32)
        gsrb.check(ctx.scan(d, o, n), "scan")
        ctx.check_status("scan")
        ref = np.concatenate([[0.0], np.cumsum(a[:-1].astype(np.float64))])
        got = o.download()
        assert np.all(np.isinf(got) == np.isinf(ref)) and not np.any(np.isnan(got))
        fin = np.isfinite(ref)
        # FP32 within a warp's 128 elements (seven roundings), FP64 between, one rounding of the result
        assert np.all(np.abs(got[fin] - ref[fin]) <= 8 * 2.0**-24 * ref[fin])
