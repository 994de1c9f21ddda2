"""PageRank with a damping of 0: every source pushes zeros, which leaves the ranks
at their initial residual, and its edges count as relaxed like any others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["sync", "async"])
@pytest.mark.parametrize("resident", [0, 9000])
@pytest.mark.parametrize("policy", ["plain", "learned"])
def test_zero_pushes_are_counted(gpu, mode, resident, policy):
    g = gpu.Graph.rmat(12, 10, seed=2)
    eng = gpu.Engine(g, budget_bytes=resident and 36 * g.n + 96 * 1024 + resident * 8)
    eng.set_policy(policy)
    v, st = eng.run("pr", mode, pr_damping=0.0)
    assert st["relaxed_edges"] == g.m and st["global_iterations"] == 1
    assert np.all(v == np.float32(0.15))
