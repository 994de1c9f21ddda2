"""The partition plan that a run uses is made by the last CTA of the generate's
write pass, not by the step API's planner kernel: the trace of the first global
iteration against the host planner, for one partition, some, more than the
control block reports and more than the planning CTA has threads."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(gpu, g, spare):
    for kb in range(4700, 6000, 20):  # the smallest budget that fits, in 20 KB steps
        try:
            gpu.Engine(g, budget_bytes=kb * 1024).close()
            return gpu.Engine(g, budget_bytes=(kb + spare * 8) * 1024)
        except gpu.SgwError:
            pass


@pytest.mark.parametrize("mode", ["sync", "async"])
@pytest.mark.parametrize("spare,lo,hi", [(0, 257, 2000), (40, 17, 256), (400, 2, 16), (9000, 1, 1)])
def test_plan_of_the_first_iteration(gpu, orc, spare, lo, hi, mode):
    g = gpu.Graph.rmat(18, 16, seed=19)
    eng = _engine(gpu, g, spare)
    cap = eng.max_partition_size()
    eng.state_init("cc", mode)
    nodes, ptr = eng.read_active()
    fr, sz = gpu.plan_partitions(ptr, cap)
    assert lo <= len(fr) <= hi
    eng.trace_enable(True)
    vals, st = eng.run("cc", mode)
    assert np.array_equal(vals, orc.run("cc", g.node_pointer, g.edges, 0))
    cnt = C.c_uint64()
    gpu.check(gpu.lib().sgw_trace_count(eng.h, C.byref(cnt)), "trace")
    rec = np.zeros(cnt.value, gpu.TRACE_REC)
    gpu.check(gpu.lib().sgw_trace_read(eng.h, rec.ctypes.data, cnt.value, C.byref(cnt)), "trace")
    assert len(rec) == st["partitions"]
    one = rec[rec["global_iteration"] == 1]
    assert (one["num_partitions"] == len(fr)).all() and len(one) == len(fr)
    assert one["partition"].tolist() == list(range(len(fr)))
    assert np.array_equal(one["first_vertex"], nodes[fr]) and np.array_equal(one["active_nodes"], sz)
    assert np.array_equal(one["active_edges"], ptr[fr + sz].astype(np.uint64) - ptr[fr])
    for it in range(2, int(rec["global_iteration"].max()) + 1):  # later plans: whole queues, within the buffer
        r = rec[rec["global_iteration"] == it]
        assert len(r) == r["num_partitions"][0]
        assert r["active_nodes"].sum() == r["iteration_active_nodes"][0]
        assert r["active_edges"].sum() == r["iteration_active_edges"][0]
        assert ((r["active_edges"] <= cap) | (r["active_nodes"] == 1)).all()
        assert (np.diff(r["first_vertex"].astype(np.int64)) > 0).all()
        # greedy: a partition and its successor's first vertex do not fit together
        deg = g.out_degree()
        assert (r["active_edges"][:-1] + deg[r["first_vertex"][1:]] > cap).all()
