"""The work units of a batch's frontier are counted in the low 32 bits of a
counter whose high word counts its rows: no graph may carry into the rows."""
import numpy as np
import pytest


def _units(deg, unit):
    return int(np.sum(np.where(deg > 0, 1 + -(-deg // unit), 0)))


@pytest.mark.parametrize("n,m", [(1 << 16, 1 << 20), (1 << 27, (1 << 35) - (1 << 31) - 1), (1 << 27, (1 << 35) - (1 << 31)),
                                 (1 << 27, 34_200_000_000), (1 << 28, 1 << 36), (1_800_000_000, 4_000_000_000)])
def test_unit_counter_holds_the_whole_graph(native, n, m):
    """A full frontier: even with every row one edge past a whole unit, which
    makes the most units for its edges, the count stays below 2^32."""
    unit = native.lib().sgw_batch_unit_edges(n, m)
    rows = min(n, m)
    most = rows + (m - rows) // unit + rows  # a row's own unit, its whole ones, its started one
    assert most < 1 << 32
    assert unit == (8 if 2 * n + m // 8 < 1 << 32 else 64)


def test_bound_against_counted_units(native):
    rng = np.random.default_rng(1)
    for _ in range(200):
        deg = (rng.pareto(1.0, 300) * rng.integers(1, 40)).astype(np.int64)
        for unit in (8, 64):
            assert _units(deg, unit) <= 2 * len(deg) + int(deg.sum()) // unit


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [32, 64])
def test_wide_units(gpu, orc, lanes):
    """The units of 64 edges on graphs that the oracle can answer: rows shorter
    than a unit, of whole units, one edge past them, and hubs."""
    rng = np.random.default_rng(5)
    n = 4001
    deg = rng.choice([0, 1, 7, 8, 9, 63, 64, 65, 128, 129], n)
    deg[[3, 2000]] = 3900
    npt = np.zeros(n + 1, np.uint32)
    npt[1:] = np.cumsum(deg)
    dst = np.concatenate([rng.choice(n, d, replace=False) for d in deg]).astype(np.uint32)
    e = np.stack([dst, rng.integers(1, 64, len(dst)).astype(np.uint32)], 1)
    g = gpu.Graph.from_csr(npt, e, True)
    src = rng.integers(0, n, lanes - 3).astype(np.uint32)
    for flags in (gpu.OPT_BATCH_PERSISTENT, gpu.OPT_BATCH_GRAPH):
        b = gpu.Batch(g, lanes=lanes, flags=flags | gpu.OPT_BATCH_WIDE_UNITS)
        for algo in ("bfs", "sssp"):
            out, _ = b.run(algo, src)
            edges = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
            for i, s in enumerate(src):
                assert np.array_equal(out[i], orc.run(algo, g.node_pointer, edges, int(s))), (algo, flags, i)
        b.close()
