"""Performance cases: what a program that uses the library has it do.

Reductions, scans, segment batches, grid barriers and graph traversals, each
through the Python binding's public calls and, unless the case says otherwise,
with the library's default launch configuration, from the smallest calls (launch
latency) to the sizes of the benchmark plan (2^28-element scans, R-MAT scale 22,
the 2048 x 2048 grid).  listed() are fixed cases, draw() samples more from the
same ranges, run() is one pass of a prepared case.
"""
import importlib
import math

import numpy as np
import torch

gsrb = importlib.import_module("tpds22-artifact_b200.gsrb")

DEV = "cuda"
INF = 2**31 - 1
ALPHA = 0.85

_ctx = None


def _context():
    """The program's one context (a program keeps it for its whole life)."""
    global _ctx
    if _ctx is None:
        _ctx = gsrb.Context(0)
    return _ctx


def listed():
    return [
        # a sum inside a host loop: launch and fixed costs are everything
        {"name": "reduce_small", "kind": "reduce", "n": 4099},
        # the plan's reduction: 2^24 values in [0, 127], 148 x 2 x 256 threads
        {"name": "reduce_16m", "kind": "reduce", "n": 1 << 24, "ctas": 2, "threads": 256},
        # the plan's integer scan: 2^28 values in [0, 15]
        {"name": "scan_u32_256m", "kind": "scan_u32", "n": 1 << 28},
        # an ordinary FP32 scan of a ragged length
        {"name": "scan_f32_3m", "kind": "scan_f32", "n": 3_000_001},
        # the plan's segment batch: 64 uneven segments scanned in one launch
        {"name": "segments_scan_64", "kind": "seg_scan_u32", "k": 64, "lo": 10.0, "hi": 22.0, "lens": 7},
        # the grid barrier itself at full residency (148 x 8 x 256 threads)
        {"name": "barrier_k8", "kind": "barrier", "ctas": 8, "episodes": 1000, "fma": 0},
        # power-law graph, few fat levels
        {"name": "bfs_rmat22", "kind": "bfs", "graph": "rmat", "scale": 22, "factor": 16},
        # mesh / road-like graph, thousands of thin levels
        {"name": "bfs_grid2048", "kind": "bfs", "graph": "grid", "width": 2048, "height": 2048},
        # weighted mesh: thousands of thin relax rounds
        {"name": "sssp_grid2048", "kind": "sssp", "graph": "grid", "width": 2048, "height": 2048, "delta": 10000},
        # many power-law graphs of uneven sizes in one launch
        {"name": "batch_sssp_16", "kind": "batch_sssp", "k": 16, "lo": 13, "hi": 17, "delta": 10000},
        # the plan's pull PageRank, 50 iterations
        {"name": "pagerank_rmat20", "kind": "pagerank", "graph": "rmat", "scale": 20, "factor": 16, "iters": 50},
        # the reference harness's PageRank: residual pushes until nothing exceeds 1e-6
        {"name": "pagerank_residual_rmat20", "kind": "pr_residual", "graph": "rmat", "scale": 20, "factor": 16},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_scale, max_side):
    if rng.random() < 0.5:
        return {"graph": "rmat", "scale": rng.randint(10, max_scale), "factor": rng.randint(6, 24)}
    return {"graph": "grid", "width": _log_uniform(rng, 24, max_side), "height": _log_uniform(rng, 24, max_side)}


def draw(rng):
    kind = rng.choice(["reduce", "scan_u32", "scan_f32", "seg_reduce", "seg_scan_u32", "seg_scan_f32", "barrier",
                       "bfs", "sssp", "batch_bfs", "batch_sssp", "pagerank", "pr_residual"])
    c = {"kind": kind}
    if kind == "reduce":
        c["n"] = _log_uniform(rng, 500, 1 << 28)
        if rng.random() < 0.5:  # the plan's launch shape; otherwise the default
            c.update(ctas=2, threads=256)
    elif kind in ("scan_u32", "scan_f32"):
        c["n"] = _log_uniform(rng, 500, 1 << 28)
    elif kind in ("seg_reduce", "seg_scan_u32", "seg_scan_f32"):
        lo = rng.uniform(4.0, 14.0)
        c.update(k=rng.randint(2, 127), lo=round(lo, 2), hi=round(lo + rng.uniform(1.0, 8.0), 2),
                 lens=rng.randint(1, 10**6))
    elif kind == "barrier":
        c.update(ctas=rng.choice([1, 2, 4, 8]), episodes=_log_uniform(rng, 50, 1000), fma=rng.choice([0, 64, 1024]))
    elif kind == "bfs":
        c.update(_draw_graph(rng, 21, 1800))
    elif kind == "sssp":
        c.update(_draw_graph(rng, 20, 1400))
        c["delta"] = 10000
    elif kind in ("batch_bfs", "batch_sssp"):
        c.update(k=rng.randint(2, 24), lo=rng.randint(10, 12), hi=rng.randint(13, 16))
        if kind == "batch_sssp":
            c["delta"] = 10000
    elif kind == "pagerank":
        c.update(_draw_graph(rng, 20, 1400))
        c["iters"] = rng.choice([10, 20, 50])
    else:
        c.update(_draw_graph(rng, 19, 700))
    return c


# ---- inputs, made on the GPU from the seed alone ------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2 + 1)


def _csr_of_pairs(n, u, v, wlo, whi, gen):
    """CSR (row int32[n+1], dst int32[m], weight int32[m]) of the undirected graph with these vertex pairs:
    no self loops, no duplicates, rows sorted, one weight per undirected edge."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = torch.unique(torch.minimum(u, v) * n + torch.maximum(u, v))
    w = torch.randint(wlo, whi + 1, (key.numel(),), generator=gen, device=DEV, dtype=torch.int32)
    u, v = key // n, key % n
    both, order = torch.sort(torch.cat([u * n + v, v * n + u]))
    w = torch.cat([w, w])[order]
    row = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row[1:] = torch.cumsum(torch.bincount(both // n, minlength=n), 0)
    return row.to(torch.int32), (both % n).to(torch.int32), w


def _rmat(scale, factor, gen, wlo=1, whi=255):
    """R-MAT, `factor` edges per vertex, a = 0.57, b = c = 0.19, symmetrised (vertex 0 has the most edges)."""
    n, e = 1 << scale, factor << scale
    u = torch.zeros(e, dtype=torch.int64, device=DEV)
    v = torch.zeros(e, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        r = torch.rand(e, generator=gen, device=DEV)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return (n,) + _csr_of_pairs(n, u, v, wlo, whi, gen)


def _grid(width, height, gen, wlo=1, whi=1000):
    """width x height grid, 4 neighbours."""
    n = width * height
    ids = torch.arange(n, dtype=torch.int64, device=DEV).reshape(height, width)
    u = torch.cat([ids[:, :-1].reshape(-1), ids[:-1, :].reshape(-1)])
    v = torch.cat([ids[:, 1:].reshape(-1), ids[1:, :].reshape(-1)])
    return (n,) + _csr_of_pairs(n, u, v, wlo, whi, gen)


def _graph(case, seed):
    """(n, row, dst, weights, source)"""
    gen = _gen(seed)
    if case["graph"] == "rmat":
        n, row, dst, w = _rmat(case["scale"], case["factor"], gen)
        return n, row, dst, w, 0  # vertex 0, the hub
    n, row, dst, w = _grid(case["width"], case["height"], gen)
    # a source near a corner, so that the wave crosses the grid
    y = int(torch.randint(0, max(1, case["height"] // 64), (1,), generator=gen, device=DEV))
    x = int(torch.randint(0, max(1, case["width"] // 64), (1,), generator=gen, device=DEV))
    return n, row, dst, w, y * case["width"] + x


def _host_graph(row, dst, w):
    return gsrb.Graph(row.cpu().numpy().view(np.uint32), dst.cpu().numpy().view(np.uint32), w.cpu().numpy())


def _offsets(case):
    """Offsets of k segments of 2^U(lo, hi) elements; the lengths are part of the case."""
    rng = np.random.default_rng(case["lens"])
    lens = np.exp2(rng.uniform(case["lo"], case["hi"], case["k"])).astype(np.uint64)
    return np.concatenate([np.zeros(1, np.uint64), np.cumsum(lens, dtype=np.uint64)])


def _batch_scales(case):
    """The instances' R-MAT scales, spread over [lo, hi]."""
    k, lo, hi = case["k"], case["lo"], case["hi"]
    return [lo + (i * (hi - lo + 1)) // k for i in range(k)]


def _values(kind, n, gen):
    if kind.endswith("f32"):
        return torch.rand(n, generator=gen, device=DEV)
    top = 128 if "reduce" in kind else 16
    return torch.randint(0, top, (n,), generator=gen, device=DEV, dtype=torch.int32)


def _seeds(case, seed):
    """One FP32 state per thread of a barrier benchmark launch."""
    return torch.rand(_context().num_sms * case["ctas"] * 256, generator=_gen(seed), device=DEV)


def _ref(t, dtype):
    """A torch tensor's device address, as the binding's calls take it."""
    return gsrb.ElementRef(t.data_ptr(), dtype)


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = {"kind": kind, "ctx": ctx, "case": case}
    if kind in ("reduce", "scan_u32", "scan_f32"):
        s["in"] = _values(kind, case["n"], _gen(seed))
        s["n"] = case["n"]
        s["cfg"] = None
        if kind == "reduce":
            s["out"] = torch.zeros(1, dtype=torch.int64, device=DEV)
            if "ctas" in case:
                s["cfg"] = gsrb.cfg(variant=gsrb.BAR_FANOUT, ctas_per_sm=case["ctas"], threads=case["threads"])
        else:
            s["out"] = torch.empty_like(s["in"])
        dt = np.float32 if kind == "scan_f32" else np.int32
        s["din"], s["dout"] = _ref(s["in"], dt), _ref(s["out"], dt)
    elif kind.startswith("seg_"):
        s["off"] = _offsets(case)
        s["in"] = _values(kind, int(s["off"][-1]), _gen(seed))
        if kind == "seg_reduce":
            s["out"] = torch.zeros(case["k"], dtype=torch.int64, device=DEV)
        else:
            s["out"] = torch.empty_like(s["in"])
        dt = np.float32 if kind == "seg_scan_f32" else np.int32
        s["din"], s["dout"] = _ref(s["in"], dt), _ref(s["out"], dt)
    elif kind == "barrier":
        s["cfg"] = gsrb.cfg(variant=gsrb.BAR_FANOUT, ctas_per_sm=case["ctas"], threads=256)
        s["sink"] = _seeds(case, seed)
        s["count"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        s["dsink"], s["dcount"] = _ref(s["sink"], np.float32), _ref(s["count"], np.uint32)
    elif kind.startswith("batch_"):
        gen = _gen(seed)
        s["graphs"] = []
        for scale in _batch_scales(case):
            _, row, dst, w = _rmat(scale, 16, gen)
            s["graphs"].append(ctx.graph(_host_graph(row, dst, w)))
        s["batch"] = gsrb.Batch(ctx, s["graphs"])
        s["srcs"] = [0] * case["k"]
        s["out"] = [torch.empty(g.n, dtype=torch.int32, device=DEV) for g in s["graphs"]]
        s["dout"] = [_ref(t, np.int32) for t in s["out"]]
    else:
        n, row, dst, w, s["src"] = _graph(case, seed)
        s["graph"] = ctx.graph(_host_graph(row, dst, w))
        s["out"] = torch.empty(n, dtype=torch.float32 if kind in ("pagerank", "pr_residual") else torch.int32,
                               device=DEV)
        s["dout"] = _ref(s["out"], np.float32)
    torch.cuda.synchronize()  # the context works on a stream of its own
    return s


def run(s):
    ctx, kind, case = s["ctx"], s["kind"], s["case"]
    if kind == "reduce":
        gsrb.check(ctx.reduce_i32(s["din"], s["n"], s["dout"], s["cfg"]), kind)
    elif kind in ("scan_u32", "scan_f32"):
        gsrb.check(ctx.scan(s["din"], s["dout"], s["n"]), kind)
    elif kind == "seg_reduce":
        gsrb.check(ctx.reduce_i32_segments(s["din"], s["off"], s["dout"]), kind)
    elif kind in ("seg_scan_u32", "seg_scan_f32"):
        gsrb.check(ctx.scan_segments(s["din"], s["dout"], s["off"]), kind)
    elif kind == "barrier":
        # the sink holds the threads' FMA state and the count the completed episodes; both go on from pass to pass
        gsrb.check(ctx.barrier_bench(s["cfg"], case["episodes"], case["fma"], s["dsink"], s["dcount"]), kind)
        return {"sink": s["sink"], "count": s["count"]}
    elif kind == "bfs":
        gsrb.check(s["graph"].bfs(s["src"], s["dout"])[0], kind)
    elif kind == "sssp":
        gsrb.check(s["graph"].sssp(s["src"], s["dout"], case["delta"])[0], kind)
    elif kind == "batch_bfs":
        gsrb.check(s["batch"].bfs(s["srcs"], s["dout"]), kind)
        gsrb.check(s["batch"].stats()[0], kind)  # a program reads every instance's status before it calls again
    elif kind == "batch_sssp":
        gsrb.check(s["batch"].sssp(s["srcs"], s["dout"], case["delta"]), kind)
        gsrb.check(s["batch"].stats()[0], kind)
    elif kind == "pagerank":
        gsrb.check(s["graph"].pagerank(s["dout"], ALPHA, case["iters"])[0], kind)
    else:
        gsrb.check(s["graph"].pagerank_residual(s["dout"], ALPHA, 1e-6)[0], kind)
    return s["out"]


# ---- what a pass cannot do without ---------------------------------------------------

def _size(case):
    """(vertices, directed edges) of a case's graph; R-MAT edges after duplicates, about."""
    if case["graph"] == "rmat":
        return _rmat_size(case["scale"], case["factor"])
    w, h = case["width"], case["height"]
    return w * h, 2 * ((w - 1) * h + w * (h - 1))


def _rmat_size(scale, factor):
    # about the share of the directed edges left without duplicates and self loops
    return 1 << scale, int(2 * (factor << scale) * min(0.97, 0.76 + 0.016 * (scale - 10)))


def work(case):
    kind = case["kind"]
    if kind == "reduce":
        return {"bytes": 4 * case["n"] + 8, "flops": case["n"]}
    if kind in ("scan_u32", "scan_f32"):
        return {"bytes": 8 * case["n"], "flops": case["n"]}
    if kind.startswith("seg_"):
        n = int(_offsets(case)[-1])
        return {"bytes": 4 * n if kind == "seg_reduce" else 8 * n, "flops": n}
    if kind == "barrier":
        threads = 148 * case["ctas"] * 256
        return {"bytes": 8 * threads, "flops": 2 * threads * case["fma"] * case["episodes"]}
    if kind.startswith("batch_"):
        total = 0
        for scale in _batch_scales(case):
            n, m = _rmat_size(scale, 16)
            total += 8 * n + (4 if kind == "batch_bfs" else 8) * m
        return {"bytes": total, "flops": 0}
    n, m = _size(case)
    if kind == "bfs":
        return {"bytes": 8 * n + 4 * m, "flops": 0}
    if kind == "sssp":
        return {"bytes": 8 * n + 8 * m, "flops": m}
    if kind == "pagerank":
        # every iteration sums every edge; rows, edges and ranks cross memory at least once
        return {"bytes": 8 * n + 4 * m, "flops": 2 * m * case["iters"]}
    return {"bytes": 8 * n + 4 * m, "flops": 2 * m}


# ---- 64-bit results of the floating-point outputs ------------------------------------

def _exclusive_f64(x):
    y = torch.zeros(x.numel(), dtype=torch.float64, device=DEV)
    if x.numel() > 1:
        y[1:] = torch.cumsum(x[:-1].double(), 0)
    return y


def _pagerank_f64(n, row, dst, iters):
    deg = (row[1:] - row[:-1]).double()
    src = torch.repeat_interleave(torch.arange(n, device=DEV), (row[1:] - row[:-1]).long())
    x = torch.full((n,), 1.0 - ALPHA, dtype=torch.float64, device=DEV)
    for _ in range(iters):
        share = torch.where(deg > 0, x / deg.clamp(min=1), torch.zeros_like(x))
        x = (1.0 - ALPHA) + ALPHA * torch.zeros_like(x).index_add_(0, src, share[dst.long()])
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "scan_f32":
        return _exclusive_f64(_values(kind, case["n"], _gen(seed)))
    if kind == "seg_scan_f32":
        off = _offsets(case).astype(np.int64)
        x = _values(kind, int(off[-1]), _gen(seed))
        return torch.cat([_exclusive_f64(x[a:b]) for a, b in zip(off[:-1], off[1:])])
    if kind == "barrier" and case["fma"] == 0:
        # no FMAs between the episodes: every thread's state stays what it was
        return {"sink": _seeds(case, seed).double(), "count": None}
    if kind == "pagerank":
        n, row, dst, _, _ = _graph(case, seed)
        return _pagerank_f64(n, row, dst, case["iters"])
    if kind == "pr_residual":
        n, row, dst, _, _ = _graph(case, seed)
        return _pagerank_f64(n, row, dst, 160)  # the fixed point the residual pushes approach: 0.85^160 < 1e-11
    return None
