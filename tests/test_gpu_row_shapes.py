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
