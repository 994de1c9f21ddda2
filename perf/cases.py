"""The calls whose speed this framework is measured by.

A case is one pass of a user's program through the public entry points of
subway_gb300.native (or, for the compaction step, of the C ABI):

  query       one BFS / SSSP / SSWP / CC / PageRank run of an engine that a
              service keeps, under a device-memory budget: host copy of the
              edges, partitions or learned schedule, answer in host memory
  one_query   what the drop-in apps do per process: create an engine that
              reads the graph's records in place, run one query, destroy it
  batch       up to 64 BFS / SSSP queries over a graph held in HBM
  compaction  the frontier compaction on caller-owned device arrays

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05) and Erdos-Renyi, without
self-loops and duplicates, as the library's own generators make them; they
are made on the GPU here because preparing them on the host would take most
of the measuring time.  Integer answers are exact fixpoints: they do not
depend on the order in which edges are relaxed.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from subway_gb300 import native as N
from subway_gb300 import scheduler

DEVICE = 0
RMAT_A, RMAT_B, RMAT_C = 0.57, 0.19, 0.19


# ---- cases -----------------------------------------------------------------------

def _query(name, algo, mode, n, ef, *, graph="rmat", wmax=0, resident=0.0, policy="plain", acc=0.0):
    """resident: share of the edges' transfer bytes that the budget leaves
    for edge buffers beside the vertex state (0: no budget, the whole GPU)."""
    c = {"kind": "query", "algo": algo, "mode": mode, "graph": graph, "n": n, "ef": ef, "wmax": wmax,
         "resident": resident, "policy": policy, "acc": acc}
    return {"name": name, **c} if name else c


def _one_query(name, algo, mode, log2n, ef, wmax, resident, policy):
    c = {"kind": "one_query", "algo": algo, "mode": mode, "log2n": log2n, "ef": ef, "wmax": wmax,
         "resident": resident, "policy": policy}
    return {"name": name, **c} if name else c


def _batch(name, algo, n, ef, queries, lanes, answers, wmax):
    c = {"kind": "batch", "algo": algo, "n": n, "ef": ef, "queries": queries, "lanes": lanes,
         "answers": answers, "wmax": wmax}
    return {"name": name, **c} if name else c


def _compaction(name, n, ef, active):
    c = {"kind": "compaction", "n": n, "ef": ef, "active": active}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest query in use: a 1 M-edge graph that fits the GPU, where launches and
        # host round trips count (BFS from one source of R-MAT 2^16)
        _query("bfs_sync_64k", "bfs", "sync", 1 << 16, 16),
        # the flagship: weighted SSSP on a graph far larger than the budget, learned schedule;
        # the budget leaves as small a share of the edges in HBM as 8 GB does of R-MAT 2^28,
        # and the weights do not pack beside the vertex ids, as there
        _query("sssp_async_32m_learned", "sssp", "async", 1 << 25, 16, wmax=255, resident=0.15, policy="learned"),
        # learned schedule with a whole range resident (three buffers hold most of the edges)
        _query("bfs_async_4m_learned", "bfs", "async", 1 << 22, 16, resident=0.67, policy="learned"),
        # the reference's schedule, many partitions, no hubs, a ragged vertex count
        _query("sssp_async_er_3m", "sssp", "async", 3_000_017, 12, graph="er", wmax=64, resident=0.5),
        # connected components of an undirected graph: every vertex starts active
        _query("cc_sync_2m_sym", "cc", "sync", 1 << 21, 8, graph="sym", resident=0.5),
        # widest paths with weights that fit neither the packed word nor a byte (8-byte
        # records), no budget
        _query("sswp_async_1m_records", "sswp", "async", 1_300_003, 16, wmax=1 << 20),
        # PageRank at the reference's default tolerance, out of memory, and to a tight one in memory
        _query("pr_sync_1m", "pr", "sync", 1 << 20, 16, resident=0.5, acc=0.01),
        _query("pr_async_128k_tight", "pr", "async", 131_101, 16, acc=1e-6),
        # a drop-in app's query: engine created, run and destroyed
        _one_query("one_query_sssp_2m", "sssp", "async", 21, 16, 64, 0.4, "learned"),
        # a query server's batches: a full one of BFS with 16-bit answers, a half one of SSSP
        _batch("batch_bfs_64x1m", "bfs", 1 << 20, 16, 64, 64, "u16", 0),
        _batch("batch_sssp_32x256k", "sssp", 1 << 18, 16, 32, 64, "u32", 64),
        # the compaction step of a host program that owns its arrays, ragged vertex count
        _compaction("compaction_17m", 16_777_259, 16, 0.25),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["query", "pr", "one_query", "batch", "compaction"], [50, 15, 10, 15, 10])[0]
    if kind == "query":
        algo = rng.choice(["bfs", "sssp", "sswp", "cc"])
        weighted = algo in ("sssp", "sswp")
        # weights that pack beside the ids, that go as a byte stream on large graphs, that need records
        wmax = rng.choice([64, 255, 1 << 20]) if weighted else 0
        graph = rng.choice(["rmat", "rmat", "er"]) if algo != "cc" else rng.choice(["rmat", "sym"])
        n = _log_uniform(rng, 1 << 13, 6_000_000)
        return _query(None, algo, rng.choice(["sync", "async"]), n, rng.randint(6, 16), graph=graph, wmax=wmax,
                      resident=rng.choice([0.0, 0.15, 0.3, 0.5, 0.67]), policy=rng.choice(["plain", "learned"]))
    if kind == "pr":
        if rng.random() < 0.5:
            return _query(None, "pr", "sync", _log_uniform(rng, 1 << 13, 1 << 21), rng.randint(6, 16),
                          resident=rng.choice([0.0, 0.3, 0.5]), acc=rng.choice([0.01, 0.001]))
        return _query(None, "pr", "async", _log_uniform(rng, 1 << 13, 1 << 18), rng.randint(6, 16),
                      resident=rng.choice([0.0, 0.5]), acc=1e-6)
    if kind == "one_query":
        algo = rng.choice(["bfs", "sssp", "cc"])
        return _one_query(None, algo, rng.choice(["sync", "async"]), rng.randint(14, 21), rng.randint(6, 16),
                          64 if algo == "sssp" else 0, rng.choice([0.0, 0.4]), rng.choice(["plain", "learned"]))
    if kind == "batch":
        algo = rng.choice(["bfs", "sssp"])
        lanes = rng.choice([32, 64])
        n = _log_uniform(rng, 1 << 13, (1 << 21) if algo == "bfs" else (1 << 19))
        return _batch(None, algo, n, rng.randint(6, 16), rng.randint(1, lanes), lanes, rng.choice(["u16", "u32"]),
                      0 if algo == "bfs" else 64)
    return _compaction(None, _log_uniform(rng, 1 << 16, 40_000_000), rng.randint(4, 16),
                       round(10 ** rng.uniform(-4, 0), 5))


# ---- inputs ----------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _pairs(kind, n, m, gen):
    """m vertex pairs of an Erdos-Renyi or R-MAT graph (pairs outside n, where
    n is no power of two, are left out)."""
    if kind == "er":
        return tuple(torch.randint(0, n, (m,), device="cuda", generator=gen) for _ in range(2))
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, device="cuda", generator=gen)
        s = r >= RMAT_A + RMAT_B
        d = ((r >= RMAT_A) & ~s) | (r >= RMAT_A + RMAT_B + RMAT_C)
        src.mul_(2).add_(s)
        dst.mul_(2).add_(d)
    if n & (n - 1):
        keep = (src < n) & (dst < n)
        src, dst = src[keep], dst[keep]
    return src, dst


def _csr(kind, n, ef, gen):
    """Node pointers and destinations on the GPU: sorted, no self-loops or duplicates."""
    src, dst = _pairs("er" if kind == "er" else "rmat", n, n * ef, gen)
    if kind == "sym":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    key = (src * n + dst)[src != dst]
    del src, dst
    key = torch.unique(key)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return off, key.remainder_(n)


def _source(off, ef, gen):
    """A vertex of at least average degree, so that the traversal reaches the core."""
    cand = torch.nonzero(off[1:] - off[:-1] >= ef).flatten()
    if cand.numel() == 0:
        return int(torch.argmax(off[1:] - off[:-1]))
    return int(cand[torch.randint(0, cand.numel(), (1,), device="cuda", generator=gen)])


def _host_graph(off, dst, wmax, gen):
    npt = off.to(torch.int32).cpu().numpy().view(np.uint32)
    if wmax:
        w = torch.randint(1, wmax + 1, (dst.numel(),), device="cuda", generator=gen)
        rec = torch.stack([dst, w], 1).to(torch.int32)
    else:
        rec = dst.to(torch.int32)
    g = N.Graph.from_csr(npt, rec.cpu().numpy().view(np.uint32), weighted=bool(wmax))
    del rec
    torch.cuda.empty_cache()
    return g


def _budget(case, g):
    if not case["resident"]:
        return 0
    n_bits, w_bits = max(1, (g.n - 1).bit_length()), case["wmax"].bit_length()
    rec = 4 if n_bits + w_bits <= 32 else 5 if case["wmax"] < 256 else 8
    if case["kind"] == "one_query" and case["wmax"]:
        rec = 8  # records read in place
    state = 36 if case["algo"] == "pr" else 18
    return int(state * g.n + 2 * 1024 * 1024 + case["resident"] * rec * g.m)


def _engine(case, g, model, flags=0):
    budget = _budget(case, g)
    learned = case["policy"] == "learned"
    buffers = N.sched_buffers(g, budget) if learned and budget else 0
    eng = N.Engine(g, budget_bytes=budget, device=DEVICE, flags=flags, num_buffers=buffers)
    if learned:
        eng.set_policy("learned", model)
    return eng


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "compaction":
        n = case["n"]
        # degrees of a power-law graph: many vertices without out-edges, a few very large
        u = torch.rand(n, device="cuda", generator=gen, dtype=torch.float64)
        deg = torch.clamp((0.25 * case["ef"] / (u + 1e-6).sqrt() - 0.3 * case["ef"]), 0, 1e5).to(torch.int64)
        off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        off[1:] = torch.cumsum(deg, 0)
        labels = [(torch.rand(n, device="cuda", generator=gen) < case["active"] / 2).to(torch.uint8)
                  for _ in range(2)]
        return {"kind": kind, "n": n, "l1": labels[0], "l2": labels[1], "off": off.to(torch.int32),
                "queue": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "ptr": torch.zeros(n + 1, dtype=torch.int32, device="cuda")}
    if kind == "one_query":
        # records read in place: a graph that the library holds, as the apps load it
        g = N.Graph.rmat(case["log2n"], case["ef"], seed=int(seed) + 1, weighted=bool(case["wmax"]),
                         wmax=case["wmax"] or 1)
        model = scheduler.load_default(DEVICE) if case["policy"] == "learned" else None
        return {"kind": kind, "case": case, "graph": g, "model": model,
                "source": int(g.pick_sources(1, seed=int(seed) + 1)[0]), "out": np.zeros(g.n, np.uint32)}
    off, dst = _csr(case.get("graph", "rmat"), case["n"], case["ef"], gen)
    if kind == "batch":
        cand = torch.nonzero(off[1:] > off[:-1]).flatten()
        pick = torch.randint(0, cand.numel(), (case["queries"],), device="cuda", generator=gen)
        sources = cand[pick].to(torch.int32).cpu().numpy().view(np.uint32)
        g = _host_graph(off, dst, case["wmax"], gen)
        # answers land in pinned memory that the server keeps
        t = torch.int16 if case["answers"] == "u16" else torch.int32
        out = torch.zeros((case["queries"], g.n), dtype=t, pin_memory=True).numpy()
        return {"kind": kind, "case": case, "graph": g, "sources": sources, "out": out,
                "batch": N.Batch(g, lanes=case["lanes"], device=DEVICE)}
    source = _source(off, case["ef"], gen)
    g = _host_graph(off, dst, case["wmax"], gen)
    del off, dst
    torch.cuda.empty_cache()
    model = scheduler.load_default(DEVICE) if case["policy"] == "learned" else None
    out = np.zeros(g.n, np.float32 if case["algo"] == "pr" else np.uint32)
    return {"kind": kind, "case": case, "graph": g, "source": source, "out": out, "model": model,
            "engine": _engine(case, g, model)}


# ---- one pass --------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "query":
        case, extra = state["case"], {}
        if case["algo"] == "pr":
            extra["pr_acc"] = case["acc"]
        out, _ = state["engine"].run(case["algo"], case["mode"], state["source"], out=state["out"], **extra)
        return out if case["algo"] == "pr" else out.view(np.int32)
    if kind == "one_query":
        case = state["case"]
        eng = _engine(case, state["graph"], state["model"], N.OPT_GRAPH_IN_PLACE | N.OPT_PAGEABLE_COPY)
        out, _ = eng.run(case["algo"], case["mode"], state["source"], out=state["out"])
        eng.close()
        return out.view(np.int32)
    if kind == "batch":
        case = state["case"]
        out, _ = state["batch"].run(case["algo"], state["sources"], out=state["out"], answers=case["answers"])
        return out
    count, edges = C.c_uint32(), C.c_uint64()
    # consume = 0, the form of the asynchronous loops: queued vertices keep their labels
    st = N.lib().sgw_generate_noalloc(state["l1"].data_ptr(), state["l2"].data_ptr(), state["off"].data_ptr(),
                                      state["n"], 0, state["queue"].data_ptr(), state["ptr"].data_ptr(),
                                      C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(count),
                                      C.byref(edges))
    N.check(st, "sgw_generate_noalloc")
    # the entries past the count are the zeros that prepare() left there
    return {"count": count.value, "edges": edges.value, "queue": state["queue"], "ptr": state["ptr"],
            "label1": state["l1"], "label2": state["l2"]}


def work(case):
    """What a pass cannot do without: each edge record that the traversal
    needs read once, each answer written once, one relaxation (an addition and
    a comparison) per edge and query."""
    kind = case["kind"]
    n = (1 << case["log2n"]) if kind == "one_query" else case["n"]
    if kind == "compaction":
        # labels and, of the active vertices, pointers in; queue and pointers out
        return {"bytes": 2 * n + 16 * case["active"] * n, "flops": 0}
    m = n * case["ef"] * (2 if case.get("graph") == "sym" else 1)
    if kind == "batch":
        answer = 2 if case["answers"] == "u16" else 4
        return {"bytes": 4 * n + 4 * m + answer * n * case["queries"], "flops": 2 * m * case["queries"]}
    weighted = case["algo"] in ("sssp", "sswp")
    rec = 4
    if weighted:
        n_bits, w_bits = max(1, (n - 1).bit_length()), case["wmax"].bit_length()
        rec = 4 if n_bits + w_bits <= 32 else 5 if case["wmax"] < 256 else 8
    return {"bytes": 4 * n + rec * m + 4 * n, "flops": 2 * m}


def exact(case, seed):
    """PageRank's bulk-synchronous rounds in 64 bits; None elsewhere: integer
    answers have no rounding, and an asynchronous PageRank's value depends
    (within its tolerance) on the order its rounds take."""
    if case["kind"] != "query" or case["algo"] != "pr" or case["mode"] != "sync":
        return None
    off, dst = _csr(case["graph"], case["n"], case["ef"], _generator(seed))
    n = case["n"]
    deg = off[1:] - off[:-1]
    src = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
    init, damping, acc = (float(np.float32(x)) for x in (0.15, 0.85, case["acc"]))
    rank = torch.zeros(n, dtype=torch.float64, device="cuda")
    delta = torch.full((n,), init, dtype=torch.float64, device="cuda")
    while True:
        active = delta > acc
        if not bool(active.any()):
            break
        moved = torch.where(active, delta, torch.zeros_like(delta))
        rank += moved
        delta -= moved
        push = torch.where(deg > 0, damping * moved / deg.clamp(min=1), torch.zeros_like(moved))
        delta.index_add_(0, dst, push[src])
        # a round ends when no vertex with out-edges is left to push
        if not bool((push != 0).any()):
            break
    return rank.cpu().numpy()
