"""Edges of the generate step: arrays that start off 16-byte boundaries, sizes
around a lane's group, a tile and a CTA's run of tiles, and the partition plan
that its last CTA makes, against the oracle's compaction and the host planner."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _noalloc(native, torch, l1, l2, off, n, consume):
    queue = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    ptr = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")
    cnt, edges = C.c_uint32(), C.c_uint64()
    torch.cuda.synchronize()
    st = native.lib().sgw_generate_noalloc(l1.data_ptr(), l2.data_ptr(), off.data_ptr(), n, consume,
                                           queue.data_ptr(), ptr.data_ptr(),
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream),
                                           C.byref(cnt), C.byref(edges))
    native.check(st, "sgw_generate_noalloc")
    c = cnt.value
    q, p = queue.cpu().numpy(), ptr.cpu().numpy()
    assert (q[c:] == -1).all() and (p[c + 1:] == -1).all()  # nothing written past the count
    return q[:c].view(np.uint32), p[: c + 1].view(np.uint32), edges.value


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4097, 3 * 4096 + 16, 700 * 4096 + 5])
@pytest.mark.parametrize("shift", [(0, 0, 0), (1, 0, 0), (0, 3, 0), (0, 0, 1), (8, 8, 2)])
def test_noalloc_alignment_and_sizes(gpu, orc, n, shift):
    torch = pytest.importorskip("torch")
    if n > 100_000 and shift not in ((0, 0, 0), (8, 8, 2)):
        pytest.skip("the large size runs aligned and unaligned once each")
    rng = np.random.default_rng(n + 7)
    deg = rng.integers(0, 4, n).astype(np.uint32)
    off = np.zeros(n + 1, np.uint32)
    off[1:] = np.cumsum(deg)
    for consume in (0, 1):
        l1 = (rng.random(n) < 0.2).astype(np.uint8)
        l2 = (rng.random(n) < 0.1).astype(np.uint8)
        dl1 = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")
        dl2 = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")
        dof = torch.zeros(n + 5, dtype=torch.int32, device="cuda")
        a, b, c = shift
        dl1[a:a + n] = torch.from_numpy(l1).cuda()
        dl2[b:b + n] = torch.from_numpy(l2).cuda()
        dof[c:c + n + 1] = torch.from_numpy(off.view(np.int32)).cuda()
        q, p, e = _noalloc(gpu, torch, dl1[a:], dl2[b:], dof[c:], n, consume)
        q_all, p_all = orc.generate(l1, l2, deg)
        keep = deg[q_all] > 0
        assert np.array_equal(q, q_all[keep]) and np.array_equal(p[:-1], p_all[:-1][keep])
        assert p[-1] == p_all[-1] == e
        active = (l1 | l2) != 0
        cleared = active & ((deg == 0) | bool(consume))
        for d, s, ref in ((dl1, a, l1), (dl2, b, l2)):
            got = d.cpu().numpy()
            assert np.array_equal(got[s:s + n], np.where(cleared, 0, ref))
            assert not got[:s].any() and not got[s + n:].any()


@pytest.mark.parametrize("spare,lo,hi", [(0, 257, 2000), (40, 17, 256), (400, 2, 16), (9000, 1, 1)])
def test_partition_plan(gpu, spare, lo, hi):
    """One partition, some, more than the control block reports and more than
    the planning CTA has threads: from / size / edges equal the host planner's."""
    g = gpu.Graph.rmat(18, 16, seed=19)
    base = 0
    for kb in range(4700, 6000, 20):  # the smallest budget that fits, in 20 KB steps
        try:
            gpu.Engine(g, budget_bytes=kb * 1024).close()
            base = kb
            break
        except gpu.SgwError:
            pass
    eng = gpu.Engine(g, budget_bytes=(base + spare * 8) * 1024)
    cap = eng.max_partition_size()
    eng.state_init("cc", "sync")
    nodes, ptr = eng.read_active()
    parts = eng.partition()
    assert lo <= len(parts) <= hi, (len(parts), cap, base)
    fr, sz = gpu.plan_partitions(ptr, cap)
    assert [p[0] for p in parts] == fr.tolist() and [p[2] for p in parts] == sz.tolist()
    assert [p[3] for p in parts] == [int(ptr[f + s]) - int(ptr[f]) for f, s in zip(fr, sz)]
    vals, st = eng.run("cc", "sync")  # the same plan made by the generate's last CTA
    assert st["partitions"] >= len(parts)
