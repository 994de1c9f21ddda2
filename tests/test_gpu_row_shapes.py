"""Relaxation of rows whose shapes stress the cut of the work into warps: one
row that many warps share, thousands of one-edge rows in one warp's share, rows
that end exactly at a share's edge, empty rows between full ones.  Bit-exact
against the oracle, every algorithm and mode, in memory and in partitions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(shape, n):
    """Destinations of each vertex."""
    rng = np.random.default_rng(n)
    if shape == "star":      # vertex 0 reaches all, the others have one edge back or none
        return [np.arange(1, n)] + [np.array([0] if v % 3 else []) for v in range(1, n)]
    if shape == "path":      # one edge each
        return [np.array([v + 1]) for v in range(n - 1)] + [np.array([], int)]
    if shape == "blocks":    # rows of 248 edges: with the source's own 8 units a share of 256
        k = min(248, n - 1)
        return [np.sort(rng.choice(n, k, replace=False)) if v % 2 == 0 else np.array([], int) for v in range(n)]
    # "mixed": degrees over four decades
    deg = np.minimum((rng.pareto(0.8, n) * 2).astype(int), n - 1)
    return [np.sort(rng.choice(n, d, replace=False)) for d in deg]


def _graph(gpu, shape, n, weighted):
    rows = _rows(shape, n)
    np_ = np.zeros(n + 1, np.uint32)
    np_[1:] = np.cumsum([len(r) for r in rows])
    dst = np.concatenate(rows).astype(np.uint32) if np_[-1] else np.zeros(0, np.uint32)
    if not weighted:
        return gpu.Graph.from_csr(np_, dst, False)
    w = np.random.default_rng(n + 1).integers(1, 64, len(dst)).astype(np.uint32)
    return gpu.Graph.from_csr(np_, np.stack([dst, w], 1), True)


@pytest.mark.parametrize("shape", ["star", "path", "blocks", "mixed"])
@pytest.mark.parametrize("n", [2, 33, 257, 3001])
def test_row_shapes(gpu, orc, shape, n):
    for weighted in (False, True):
        g = _graph(gpu, shape, n, weighted)
        if g.m == 0:
            continue
        budgets = [0] if n < 257 else [0, 18 * n + 72 * 1024 + 1200 * 16]
        for budget in budgets:
            eng = gpu.Engine(g, budget_bytes=budget)
            for algo in ("sssp", "sswp") if weighted else ("bfs", "cc"):
                ref = orc.run(algo, g.node_pointer, g.edges, 0)
                for mode in ("sync", "async"):
                    if shape == "path" and n > 257 and budget and mode == "async":
                        continue  # thousands of partitions of one vertex: covered by the sync form
                    vals, st = eng.run(algo, mode, 0)
                    assert np.array_equal(vals, ref), (shape, n, algo, mode, budget)
            eng.close()


@pytest.mark.parametrize("tile_degree_max", [32, 256, 5000])
def test_hub_thresholds(gpu, orc, tile_degree_max):
    """A warp tile whose edges fill several segments of its owner table, with
    and without chunk lists."""
    g = _graph(gpu, "mixed", 3001, True)
    eng = gpu.Engine(g, tile_degree_max=tile_degree_max)
    for algo in ("sssp", "sswp", "cc"):
        ref = orc.run(algo, g.node_pointer, np.ascontiguousarray(g.ends) if algo == "cc" else g.edges, 0)
        for mode in ("sync", "async"):
            vals, _ = eng.run(algo, mode, 0)
            assert np.array_equal(vals, ref), (algo, mode)


FORMS = [("packed", {}), ("split", {"flags": "OPT_SPLIT_WEIGHTS"}), ("records", {"flags": "OPT_NO_PACK"}),
         ("in_place", {"flags": "OPT_GRAPH_IN_PLACE"}), ("chunks", {"transfer_chunk_log2": 12})]


@pytest.mark.parametrize("policy", ["plain", "learned"])
@pytest.mark.parametrize("form", [f[0] for f in FORMS])
def test_sync_reads_every_transfer_form(gpu, orc, form, policy):
    """Sync passes read the host copy themselves: packed words, the split
    form's two streams, records, the graph in place, and copies cut into 4 KiB
    chunks, with rows that start at every alignment.  Integer answers are the
    oracle's; PageRank's equal the gathering form's to its FP32 rounding."""
    opts = dict(dict(FORMS)[form])
    flags = getattr(gpu, opts.pop("flags"), 0) if "flags" in opts else 0
    g = gpu.Graph.rmat(11, 9, seed=77, weighted=True, wmax=200)
    budget = 36 * g.n + 96 * 1024 + 3000 * 16
    eng = gpu.Engine(g, budget_bytes=budget, flags=flags, **opts)
    ref_eng = gpu.Engine(g, budget_bytes=budget, flags=gpu.OPT_SCALAR_GATHER)
    if policy == "learned":
        eng.set_policy("learned")
    src = int(g.pick_sources(1, seed=5)[0])
    for algo in ("bfs", "sssp", "sswp", "cc"):
        e = g.edges if algo in ("sssp", "sswp") else np.ascontiguousarray(g.ends)
        vals, st = eng.run(algo, "sync", src)
        assert np.array_equal(vals, orc.run(algo, g.node_pointer, e, src)), algo
        assert st["partitions"] > 1 and st["gather_launches"] == 0 or policy == "learned"
    a, _ = eng.run("pr", "sync", pr_acc=0.001)
    b, _ = ref_eng.run("pr", "sync", pr_acc=0.001)
    # FP64 sums in another order, cast to FP32: one unit in the last place
    assert np.max(np.abs(a.astype(np.float64) - b) / b) < 1.2e-7 * 2


@pytest.mark.parametrize("tile_degree_max", [8, 256])
def test_pagerank_async_long_and_short_rows(gpu, orc, tile_degree_max):
    """Later async passes as one launch (no row above the threshold) and as a
    claim and a push cut by edges: within the residual bound of the exact
    fixpoint, as the forms with one kernel per tile were."""
    acc = 1e-6
    g = gpu.Graph.er(3001, 24000, seed=3)
    assert 8 < int(g.out_degree().max()) < 256
    eng = gpu.Engine(g, tile_degree_max=tile_degree_max)
    v, _ = eng.run("pr", "async", pr_acc=acc)
    npt = g.node_pointer.astype(np.int64)
    deg = np.diff(npt)
    src = np.repeat(np.arange(g.n), deg)
    rank = np.full(g.n, 0.15)
    for _ in range(400):
        nxt = np.full(g.n, 0.15)
        np.add.at(nxt, g.ends, 0.85 * (rank / np.maximum(deg, 1))[src])
        rank = nxt
    # every vertex is left with a residual of at most acc, 1/0.15 of which can still arrive
    bound = (acc / 0.15) * rank + 3e-7 * rank
    assert np.all(np.abs(v - rank) <= bound)


@pytest.mark.parametrize("inner_batch", [1, 2, 8])
@pytest.mark.parametrize("max_inner", [0, 1, 2, 4, 5])
def test_async_iterations_polled(gpu, orc, inner_batch, max_inner):
    """The host follows the inner iterations through a word of mapped memory:
    caps below, at and above the launches it keeps ahead, with and without the
    trace (whose per-partition counts come from the device and add up)."""
    import ctypes as C
    g = gpu.Graph.rmat(12, 12, seed=5, weighted=True)
    eng = gpu.Engine(g, budget_bytes=18 * g.n + 96 * 1024 + 9000 * 8, inner_batch=inner_batch)
    src = int(g.pick_sources(1, seed=6)[0])
    for algo in ("sssp", "cc"):
        e = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
        ref = orc.run(algo, g.node_pointer, e, src)
        eng.trace_enable(False)
        vals, st = eng.run(algo, "async", src, max_inner=max_inner)
        assert np.array_equal(vals, ref)
        eng.trace_enable(True)
        vals, st = eng.run(algo, "async", src, max_inner=max_inner)
        assert np.array_equal(vals, ref)
        cnt = C.c_uint64()
        gpu.check(gpu.lib().sgw_trace_count(eng.h, C.byref(cnt)), "trace")
        rec = np.zeros(cnt.value, gpu.TRACE_REC)
        gpu.check(gpu.lib().sgw_trace_read(eng.h, rec.ctypes.data, cnt.value, C.byref(cnt)), "trace")
        assert len(rec) == st["partitions"] and int(rec["inner_iterations"].sum()) == st["inner_iterations"]
        if max_inner:
            assert int(rec["inner_iterations"].max()) <= max_inner


@pytest.mark.parametrize("form", [f[0] for f in FORMS])
@pytest.mark.parametrize("share", [0.0, 0.3, 0.8])
def test_sync_edge_cache(gpu, orc, form, share):
    """Sync runs keep the rows that fit the edge buffers: without a budget
    every record crosses the link once however often its vertex is queued, with
    one the rest is read again; the trace's bytes add up to the run's."""
    import ctypes as C
    opts = dict(dict(FORMS)[form])
    flags = getattr(gpu, opts.pop("flags"), 0) if "flags" in opts else 0
    g = gpu.Graph.rmat(13, 11, seed=31, weighted=True, wmax=200)
    budget = int(36.3 * g.n + 160 * 1024 + share * 8 * g.m) if share else 0
    eng = gpu.Engine(g, budget_bytes=budget, flags=flags, **opts)
    src = int(g.pick_sources(1, seed=5)[0])
    deg = g.out_degree()
    for algo in ("cc", "sssp", "sswp", "pr"):
        e = g.edges if algo in ("sssp", "sswp") else np.ascontiguousarray(g.ends)
        eng.trace_enable(True)
        vals, st = eng.run(algo, "sync", src)
        if algo != "pr":
            ref = orc.run(algo, g.node_pointer, e, src)
            assert np.array_equal(vals, ref), algo
        cnt = C.c_uint64()
        gpu.check(gpu.lib().sgw_trace_count(eng.h, C.byref(cnt)), "trace")
        rec = np.zeros(cnt.value, gpu.TRACE_REC)
        gpu.check(gpu.lib().sgw_trace_read(eng.h, rec.ctypes.data, cnt.value, C.byref(cnt)), "trace")
        assert int(rec["bytes_h2d"].sum()) == st["h2d_bytes"]
        eng.trace_enable(False)
        again, st2 = eng.run(algo, "sync", src)  # nothing is carried from run to run
        assert st2["h2d_bytes"] == st["h2d_bytes"] or share
        if algo != "pr":
            assert np.array_equal(again, ref)
        per_edge = {"packed": 4, "chunks": 4, "records": 8, "in_place": 8}.get(form) or (5 if algo in ("sssp", "sswp") else 4)
        assert st["h2d_bytes"] <= st["active_edges"] * per_edge
        if not share:
            once = g.m if algo in ("cc", "pr") else int(deg[ref != (4294967294 if algo == "sssp" else 0)].sum())
            assert st["h2d_bytes"] == once * per_edge, algo
            assert st["active_edges"] > once, algo  # vertices were queued again


@pytest.mark.parametrize("extra", [0, 2048, 6144, 8192, 20000])
def test_sync_cache_bits_in_small_buffers(gpu, orc, extra):
    """The edge cache's bits (n / 4 bytes) share the edge buffers: from the
    smallest accepted budget, whose buffers do not hold them, across the line."""
    g = gpu.Graph.er(30011, 60000, seed=9, weighted=True, wmax=60)
    lo, hi = 18 * g.n, 18 * g.n + (1 << 20)  # refused, accepted
    while hi - lo > 64:
        mid = (lo + hi) // 2
        try:
            gpu.Engine(g, budget_bytes=mid).close()
            hi = mid
        except gpu.SgwError:
            lo = mid
    eng = gpu.Engine(g, budget_bytes=hi + extra)
    src = int(g.pick_sources(1, seed=5)[0])
    for algo in ("cc", "sssp"):
        e = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
        vals, _ = eng.run(algo, "sync", src)
        assert np.array_equal(vals, orc.run(algo, g.node_pointer, e, src)), algo
