"""PageRank's vertex state under the smallest budgets: it holds no per-tile totals
unless an edge limit asks for them, and the gap that places the residuals is
left out where the budget has no room for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fits(gpu, g, budget, **opts):
    try:
        eng = gpu.Engine(g, budget_bytes=budget, **opts)
    except gpu.SgwError:
        return False
    try:
        eng.state_init("pr", "sync")
        return True
    except gpu.SgwError:
        return False
    finally:
        eng.close()


def _smallest(gpu, g, **opts):
    lo, hi = 32 * g.n, 64 * g.n + (1 << 20)
    assert _fits(gpu, g, hi, **opts)
    while hi - lo > 64:
        mid = (lo + hi) // 2
        if _fits(gpu, g, mid, **opts):
            hi = mid
        else:
            lo = mid
    return hi


@pytest.mark.parametrize("n", [5000, 1 << 17, 300_001])
def test_smallest_pagerank_budget(gpu, orc, n):
    g = gpu.Graph.er(n, 4 * n, seed=9)
    least = _smallest(gpu, g)
    totals = 8 * -(-n // 4096)
    assert _smallest(gpu, g, generate_edge_limit=g.m) - least >= totals // 256 * 256
    ref = None
    for budget in (least, least + 256, least + 1024, least + 4096, 0):  # without the gap, on both sides of it, with it
        eng = gpu.Engine(g, budget_bytes=budget)
        v, st = eng.run("pr", "async", pr_acc=1e-4)
        eng.close()
        # every vertex keeps at most acc of residual, of which 1/0.15 can still arrive
        ref = v if ref is None else ref
        assert np.max(np.abs(v - ref) / np.maximum(v, ref)) <= 2 * 1e-4 / 0.15
