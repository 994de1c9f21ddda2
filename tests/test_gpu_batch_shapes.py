"""Batches over graphs whose sizes end inside a frontier tile, a row's work
units or a warp's share, traversals with more levels than four level planes
hold, and frontiers on both sides of the large / small line: every lane equals
the oracle, in both forms and both widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(gpu, orc, g, algo, src, lanes, flags):
    b = gpu.Batch(g, lanes=lanes, flags=flags)
    out, _ = b.run(algo, src)
    e = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
    for i, s in enumerate(src):
        assert np.array_equal(out[i], orc.run(algo, g.node_pointer, e, int(s))), (algo, lanes, i)
    b.close()


@pytest.mark.parametrize("n", [2, 5, 1023, 1025, 5003])
@pytest.mark.parametrize("lanes", [32, 64])
def test_ragged_sizes(gpu, orc, n, lanes):
    g = gpu.Graph.er(n, 5 * n, seed=n, weighted=True, wmax=64)
    rng = np.random.default_rng(n)
    for nsrc in (1, 3, lanes):
        src = rng.integers(0, n, nsrc).astype(np.uint32)  # sources may repeat or have no out-edges
        for algo in ("bfs", "sssp"):
            for flags in (gpu.OPT_BATCH_PERSISTENT, gpu.OPT_BATCH_GRAPH):
                _check(gpu, orc, g, algo, src, lanes, flags)


@pytest.mark.parametrize("lanes", [32, 64])
@pytest.mark.parametrize("length", [15, 16, 17, 33, 300])
def test_level_planes(gpu, orc, lanes, length):
    """A path (one level per vertex): levels on both sides of the powers of
    two at which a plane is first written, 16-bit answers included."""
    npt = np.append(np.arange(length, dtype=np.uint32), np.uint32(length - 1))
    g = gpu.Graph.from_csr(npt, np.arange(1, length, dtype=np.uint32), False)
    src = np.array([0, 1, length // 2, length - 1], np.uint32)
    for flags in (gpu.OPT_BATCH_PERSISTENT, gpu.OPT_BATCH_GRAPH):
        b = gpu.Batch(g, lanes=lanes, flags=flags)
        out, _ = b.run("bfs", src)
        out16, _ = b.run("bfs", src, answers="u16")
        for i, s in enumerate(src):
            ref = orc.run("bfs", g.node_pointer, g.edges, int(s))
            assert np.array_equal(out[i], ref)
            assert np.array_equal(out16[i], np.where(ref == 4294967294, 0xFFFF, ref).astype(np.uint16))
        b.close()


def test_levels_past_16_bits(gpu):
    n = 65_600
    npt = np.append(np.arange(n, dtype=np.uint32), np.uint32(n - 1))
    g = gpu.Graph.from_csr(npt, np.arange(1, n, dtype=np.uint32), False)
    b = gpu.Batch(g, lanes=32, flags=gpu.OPT_BATCH_PERSISTENT)
    out, _ = b.run("bfs", np.array([0, 100], np.uint32))
    assert np.array_equal(out[0], np.arange(n, dtype=np.uint32))
    with pytest.raises(gpu.SgwError):
        b.run("bfs", np.array([0], np.uint32), answers="u16")
    ok, _ = b.run("bfs", np.array([100], np.uint32), answers="u16")
    assert ok[0, 100] == 0 and ok[0, n - 1] == n - 101 and ok[0, 0] == 0xFFFF


@pytest.mark.parametrize("nopack", [False, True])
def test_large_frontiers(gpu, orc, nopack):
    g = gpu.Graph.rmat(16, 16, seed=8, weighted=True, wmax=64)
    src = g.pick_sources(40, seed=2)
    fl = gpu.OPT_NO_PACK if nopack else 0
    for flags in (gpu.OPT_BATCH_PERSISTENT, gpu.OPT_BATCH_GRAPH):
        b = gpu.Batch(g, lanes=64, flags=flags | fl)
        for algo in ("bfs", "sssp"):
            out, _ = b.run(algo, src)
            e = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
            for i in (0, 7, 31, 32, 39):
                assert np.array_equal(out[i], orc.run(algo, g.node_pointer, e, int(src[i]), parallel=True)), (algo, i)
        b.close()
