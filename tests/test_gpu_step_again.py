"""The step API may process a partition again before the next generate: an async
call relaxes the sources that have been labelled since, and no others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relaxed(eng):
    return eng.stats()["relaxed_edges"]


@pytest.mark.parametrize("algo", ["sssp", "cc"])
@pytest.mark.parametrize("hub", [False, True])
def test_second_call_relaxes_what_is_left(gpu, orc, algo, hub):
    n = 20_003
    rng = np.random.default_rng(3)
    deg = rng.integers(0, 9, n)
    deg[0] = n - 1 if hub else 8
    npt = np.zeros(n + 1, np.uint32)
    npt[1:] = np.cumsum(deg)
    dst = np.concatenate([rng.choice(n, d, replace=False) for d in deg]).astype(np.uint32)
    g = gpu.Graph.from_csr(npt, np.stack([dst, rng.integers(1, 64, len(dst)).astype(np.uint32)], 1), True)
    budget = 18 * n + 72 * 1024 + 3000 * 8
    eng = gpu.Engine(g, budget_bytes=budget)
    if hub:
        assert eng.max_partition_size() < n - 1
    e = g.edges if algo == "sssp" else np.ascontiguousarray(g.ends)
    ref = orc.run(algo, g.node_pointer, e, 0)

    eng.state_init(algo, "async", 0)  # converged by the first call: nothing is left for the second
    for it in range(200):
        parts = eng.partition()
        for i in range(len(parts)):
            eng.process_partition(i)
            if hub and parts[i][3] > eng.max_partition_size():
                continue  # one pass, which may label the vertex itself
            before = _relaxed(eng)
            eng.process_partition(i)
            assert _relaxed(eng) == before, (it, i)
        if eng.generate()[0] == 0:
            break
    assert np.array_equal(eng.read_values(), ref) and _relaxed(eng) > 0

    eng.state_init(algo, "async", 0, max_inner=1)  # one pass per call: a partition is called until it is done
    for it in range(2000):
        for i in range(len(eng.partition())):
            last = -1
            for _ in range(500):
                now = _relaxed(eng)
                if now == last:
                    break
                last = now
                eng.process_partition(i)
        if eng.generate()[0] == 0:
            break
    assert np.array_equal(eng.read_values(), ref)

