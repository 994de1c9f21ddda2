"""inner_batch says how many async inner iterations are launched ahead: every
partition launches one more than that before the first report comes back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner_batch", [0, 1, 3, 4, 24])
def test_launched_ahead(gpu, orc, inner_batch):
    g = gpu.Graph.er(3001, 15000, seed=4, weighted=True, wmax=64)  # no row above tile_degree_max: one launch each
    src = int(g.pick_sources(1, seed=1)[0])
    ref = orc.run("sssp", g.node_pointer, g.edges, src)
    eng = gpu.Engine(g, inner_batch=inner_batch)
    vals, st = eng.run("sssp", "async", src)
    assert np.array_equal(vals, ref)
    ahead = inner_batch or 3
    assert st["relax_launches"] >= st["partitions"] * (1 + ahead)
    assert st["relax_launches"] <= st["inner_iterations"] + st["partitions"] * (1 + ahead)
