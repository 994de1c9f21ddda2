"""gather_bytes counts what kernels read from host memory, also where sync passes
read the host copy themselves: the rest of h2d_bytes is what DMA copies moved."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _trace(gpu, eng):
    cnt = C.c_uint64()
    gpu.check(gpu.lib().sgw_trace_count(eng.h, C.byref(cnt)), "trace")
    rec = np.zeros(cnt.value, gpu.TRACE_REC)
    gpu.check(gpu.lib().sgw_trace_read(eng.h, rec.ctypes.data, cnt.value, C.byref(cnt)), "trace")
    return rec


@pytest.mark.parametrize("algo", ["bfs", "sssp", "cc", "pr"])
@pytest.mark.parametrize("mode", ["sync", "async"])
def test_plain_runs_move_nothing_by_dma(gpu, algo, mode):
    g = gpu.Graph.rmat(12, 10, seed=6, weighted=True, wmax=64)
    eng = gpu.Engine(g, budget_bytes=36 * g.n + 96 * 1024 + 9000 * 16)
    assert int(g.out_degree().max()) <= eng.max_partition_size()  # no split vertex
    _, st = eng.run(algo, mode, int(g.pick_sources(1, seed=1)[0]))
    assert st["gather_bytes"] == st["h2d_bytes"] > 0
    assert (st["gather_launches"] == 0) == (mode == "sync")


def test_split_vertices_and_whole_ranges_are_dma(gpu):
    n = 20_001
    rng = np.random.default_rng(1)
    deg = rng.integers(0, 6, n)
    deg[7] = n - 1
    npt = np.zeros(n + 1, np.uint32)
    npt[1:] = np.cumsum(deg)
    dst = np.concatenate([rng.choice(n, d, replace=False) for d in deg]).astype(np.uint32)
    g = gpu.Graph.from_csr(npt, dst, False)
    eng = gpu.Engine(g, budget_bytes=18 * n + 72 * 1024 + 3000 * 8)
    assert eng.max_partition_size() < n - 1
    for algo in ("bfs", "cc"):
        eng.trace_enable(True)
        _, st = eng.run(algo, "sync", 7)
        rec = _trace(gpu, eng)
        assert st["h2d_bytes"] - st["gather_bytes"] == int(rec["bytes_h2d"][rec["transfer"] == 2].sum()) > 0
