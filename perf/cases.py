"""The work a user of this library has it do, as cases that can be timed.

A case names an entry point (`call`) and a graph family with its size:

  host      load_edges from host arrays, run, partition -- what start() and a
            relinked reference driver do with one graph
  device    load_edges_device (the list is already in HBM), run, partition into
            pinned memory
  pinned    load_edges_ptr from pinned host memory, run, partition into pinned
            memory: the end-to-end call of the benchmark
  steps     the reference's phase functions one by one for a level:
            modularity, one_level, renumber, induce
  unsorted  a list in arbitrary order with fractional weights (multiples of
            1/8, so that every sum is exact), each edge listed once or in both
            directions
  score     modularity_fp64 of a partition the caller brings
  batch     run_batch_device: many graphs in one packed list
  serve     Server: many requests submitted, drained and polled

Graph families are the generators of this package: R-MAT (weights 1..16), the
LFR-style power law, planted-partition SBMs (4-400 blocks, average degree
8..32, weights 1..4 unless the 10,000-vertex configuration is meant).
"""
import numpy as np
import torch

from louvaingpu_b200 import Louvain, graphgen
from louvaingpu_b200.serving import Server


MAX_LEVELS = 32    # rows of a run's level table (these graphs take 3 to 9 levels)


def listed():
    return [
        # one small graph from host lists: launches, waits and copies
        dict(name="sbm_1k_host", call="host", family="sbm", n=1000),
        # the 10,000-vertex SBM configuration (100 blocks of 100, unit weights)
        dict(name="sbm_10k_host", call="host", family="sbm_plain", n=10000),
        # an ordinary graph of an odd size, already on the device
        dict(name="sbm_120k_device", call="device", family="sbm", n=120001),
        # the power-law configuration: n = 2^20, hubs of some thousand neighbours
        dict(name="lfr_1m_device", call="device", family="lfr", n=1 << 20),
        # the largest: R-MAT, half the entries of the scale-25 configuration
        dict(name="rmat_24_device", call="device", family="rmat", scale=24, edge_factor=16, arena_gb=42),
        # end to end from pinned host memory, as the benchmark's e2e leg
        dict(name="rmat_22_pinned", call="pinned", family="rmat", scale=22, edge_factor=16),
        # phase by phase, as a driver written against the reference's functions
        dict(name="rmat_21_steps", call="steps", family="rmat", scale=21, edge_factor=16),
        # an edge list as a file holds it: any order, each edge once, real weights
        dict(name="rmat_19_unsorted", call="unsorted", family="rmat", scale=19, edge_factor=16, once=True),
        # scoring a known partition (the planted one)
        dict(name="lfr_200k_score", call="score", family="lfr", n=200003),
        # many small graphs in one call
        dict(name="batch_2048_small", call="batch", graphs=2048, n_lo=64, n_hi=2000),
        # the batched configuration's sizes (64 .. 200,000 vertices), a part of it
        dict(name="batch_128_mixed", call="batch", graphs=128, n_lo=64, n_hi=200000),
        # requests of the serving configuration's sizes, served together
        dict(name="serve_96", call="serve", graphs=96, n_lo=64, n_hi=200000, giants=2, scale=18),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["host", "device", "device", "device", "pinned", "steps", "unsorted", "score", "batch",
                       "serve"])
    if call == "host":
        return dict(call=call, family=rng.choice(["sbm", "sbm_plain"]), n=_log_int(rng, 300, 60000) | 1)
    if call == "score":
        return dict(call=call, family="lfr", n=_log_int(rng, 20000, 400000) | 1)
    if call == "batch":
        hi = _log_int(rng, 1000, 200000)
        return dict(call=call, graphs=max(32, min(_log_int(rng, 64, 2048), 6000000 // hi)), n_lo=64, n_hi=hi)
    if call == "serve":
        return dict(call=call, graphs=rng.randint(40, 120), n_lo=64, n_hi=_log_int(rng, 20000, 200000),
                    giants=rng.randint(1, 2), scale=rng.randint(16, 18))
    if call == "unsorted":
        return dict(call=call, family="rmat", scale=rng.randint(12, 19), edge_factor=rng.randint(5, 20),
                    once=rng.random() < 0.5)
    if call == "pinned":
        return dict(call=call, family="rmat", scale=rng.randint(16, 21), edge_factor=rng.randint(8, 24))
    if call == "steps":
        return dict(call=call, family="rmat", scale=rng.randint(14, 21), edge_factor=rng.randint(6, 24))
    family = rng.choice(["sbm", "sbm", "lfr", "rmat", "rmat"])
    if family == "sbm":
        return dict(call=call, family=family, n=_log_int(rng, 2000, 2000000) | 1)
    if family == "lfr":
        return dict(call=call, family=family, n=_log_int(rng, 30000, 1000000) | 1)
    return dict(call=call, family=family, scale=rng.randint(14, 23), edge_factor=rng.randint(6, 16))


class _List:
    """A symmetric, sorted edge list in device memory: src, dst and w as
    pointers, and whatever keeps them alive."""

    def __init__(self, keep, src, dst, w, n_entries, n_vertices, truth=None):
        self.keep = keep
        self.args = (src, dst, w, n_entries, n_vertices)
        self.n = n_vertices
        self.truth = truth


def _sbms(count, seed, n_lo, n_hi):
    """Parameters of `count` SBMs: sizes, blocks and degrees belong to the
    case, the edges of each graph to the seed."""
    params = graphgen.batched_sbm_params(count, seed=n_hi, n_lo=n_lo, n_hi=n_hi)
    edges = np.random.default_rng(seed).integers(0, 2**62, count)
    return [dict(p, seed=int(e)) for p, e in zip(params, edges)]


def _device_list(case, seed):
    if case["family"] == "rmat":
        g = graphgen.rmat_device(case["scale"], case["edge_factor"], seed=seed)
        return _List(g, g.src, g.dst, g.w, g.n_entries, g.n_vertices)
    if case["family"] == "sbm":
        g = graphgen.sbm_batch_device(_sbms(1, seed, case["n"], case["n"]))
        return _List(g, g.src, g.dst, g.w, g.n_entries, g.n_vertices)
    n, s, d, w = graphgen.lfr(case["n"], seed=seed)
    t = [torch.from_numpy(x).cuda() for x in (s, d, w)]
    torch.cuda.synchronize()
    return _List(t, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), len(s), n)


def _host_list(case, seed):
    if case["family"] == "sbm_plain":
        n = case["n"]
        blocks = max(2, n // 100)
        return graphgen.sbm(n, blocks, 0.1, min(1.0, 6.0 / n), 1, 1, seed)
    if case["family"] == "sbm":
        p = _sbms(1, seed, case["n"], case["n"])[0]
        return graphgen.sbm(p["n"], p["blocks"], p["p_in"], p["p_out"], 1, 4, seed)
    g = graphgen.rmat_device(case["scale"], case["edge_factor"], seed=seed)
    s, d, w = g.to_host()
    n = g.n_vertices
    g.close()
    return n, s, d, w


def _unsorted_list(case, seed):
    """(n, src, dst, w) tensors: the R-MAT edges shuffled, weights in eighths."""
    n, s, d, w = _host_list(case, seed)
    s, d, w = (torch.from_numpy(x).cuda() for x in (s, d, w))
    if case["once"]:
        up = s < d
        s, d, w = s[up], d[up], w[up]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    order = torch.randperm(len(s), generator=gen, device="cuda")
    out = (s[order].contiguous(), d[order].contiguous(), (w[order] * 0.125).contiguous())
    torch.cuda.synchronize()
    return (n, *out)


def prepare(case, seed):
    call = case["call"]
    st = {"call": call}
    if call == "batch":
        st["g"] = graphgen.sbm_batch_device(_sbms(case["graphs"], seed, case["n_lo"], case["n_hi"]))
        st["lv"] = Louvain()
        return st
    if call == "serve":
        small = graphgen.sbm_batch_device(_sbms(case["graphs"], seed, case["n_lo"], case["n_hi"]))
        giants = [graphgen.rmat_device(case["scale"], seed=seed + k) for k in range(case["giants"])]
        reqs = [small.graph_ptrs(i) for i in range(case["graphs"])]
        every = max(1, len(reqs) // (len(giants) + 1))
        for k, g in enumerate(giants):   # spread over the stream
            reqs.insert((k + 1) * every + k, (g.src, g.dst, g.w, g.n_entries, g.n_vertices))
        end = np.cumsum([r[4] for r in reqs])
        part = np.zeros(end[-1], np.int32)     # every request's partition, one after the other
        st.update(keep=(small, giants), reqs=reqs, part=part, parts=np.split(part, end[:-1]),
                  srv=Server(n_slots=4, hbm_budget=24e9, max_batch_entries=4e7))
        return st
    if call == "score":
        n, s, d, w, truth = graphgen.lfr(case["n"], seed=seed, with_truth=True)
        st["list"] = (s, d, w)
        st["truth"] = truth
        st["lv"] = Louvain()
        st["lv"].load_edges(s, d, w, n)
        return st
    if call == "host":
        st["n"], *st["list"] = _host_list(case, seed)
        st["lv"] = Louvain()
        return st
    if call == "pinned":
        st["n"], *arrays = _host_list(case, seed)
        st["list"] = [torch.from_numpy(x).pin_memory() for x in arrays]
    elif call == "unsorted":
        st["n"], *st["list"] = _unsorted_list(case, seed)
    else:
        st["list"] = _device_list(case, seed)
        st["n"] = st["list"].n
    st["part"] = torch.zeros(st["n"], dtype=torch.int32).pin_memory()
    st["lv"] = Louvain(arena_bytes=int(case.get("arena_gb", 0) * 1e9))
    return st


def _run_outputs(lv, res, part):
    level_q, sizes = np.zeros(MAX_LEVELS), np.zeros((MAX_LEVELS, 5), np.int64)
    for k in range(res.n_levels):
        x = lv.level_info(k)
        level_q[k] = x.q_level
        sizes[k] = x.n_vertices, x.n_entries, x.nnz, x.n_comms, x.passes
    return {"q": res.q_final, "communities": res.n_comms, "partition": part, "level_q": level_q, "levels": sizes}


def run(state):
    call = state["call"]
    if call == "batch":
        g = state["g"]
        r = state["lv"].run_batch_device(g.src, g.dst, g.w, g.entry_off, g.vertex_off)
        return {"partition": r.partition, "q": r.q_final, "levels": r.n_levels, "communities": r.n_comms,
                "status": r.status}
    if call == "serve":
        srv = state["srv"]
        ids = [srv.submit(*r, part_out=p) for r, p in zip(state["reqs"], state["parts"])]
        srv.drain()
        got = {r.id: r for r in srv.poll()}
        return {"partition": state["part"], "q": np.array([got[i].q_final for i in ids]),
                "communities": np.array([got[i].n_comms for i in ids]),
                "status": np.array([got[i].status for i in ids])}
    lv = state["lv"]
    if call == "score":
        return lv.modularity_fp64(state["truth"])
    if call == "host":
        lv.load_edges(*state["list"], state["n"])
        return _run_outputs(lv, lv.run(), lv.partition())
    if call == "pinned" or call == "unsorted":
        s, d, w = state["list"]
        load = lv.load_edges_ptr if call == "pinned" else lv.load_edges_device
        load(s.data_ptr(), d.data_ptr(), w.data_ptr(), len(s), state["n"])
        return _run_outputs(lv, lv.run(), lv.partition(out=state["part"]))
    lv.load_edges_device(*state["list"].args)
    if call == "device":
        return _run_outputs(lv, lv.run(), lv.partition(out=state["part"]))
    q0 = lv.modularity()                       # steps
    q1, passes = lv.one_level(q0)
    part, n_comms = lv.renumber()
    lv.induce()
    V, nnz, m = lv.csr_shape()
    return {"q": [q0, q1, lv.modularity()], "passes": passes, "communities": n_comms, "partition": part,
            "coarse": [V, nnz], "m": m}


def _size(case):
    """(vertices, entries) of a case, expected."""
    call = case["call"]
    if call in ("batch", "serve"):
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["graphs"] * (hi - lo) / np.log(hi / lo)
        e = 20.0 * n
        if call == "serve":
            n += case["giants"] * 2.0 ** case["scale"]
            e += case["giants"] * 30.0 * 2.0 ** case["scale"]
        return n, e
    if case["family"] == "rmat":
        n = 2.0 ** case["scale"]
        e = 1.9 * case["edge_factor"] * n
        return n, e / 2 if case.get("once") else e
    n = float(case["n"])
    return n, n * {"lfr": 13.66, "sbm": 20.0, "sbm_plain": 15.8}[case["family"]]


def work(case):
    # the list read once, the partition (or, for a score, nothing) written
    # once; a gain is a product and a difference for every entry of two passes
    n, e = _size(case)
    return {"bytes": 12.0 * e + 4.0 * n, "flops": 4.0 * e}


def exact(case, seed):
    """The FP64 modularity of a scored partition; the other calls' numbers
    belong to the partition the library finds."""
    if case["call"] != "score":
        return None
    _, s, d, w, truth = graphgen.lfr(case["n"], seed=seed, with_truth=True)
    a, b, w = truth[s], truth[d], w.astype(np.float64)
    comms = int(truth.max()) + 1
    strength = np.bincount(a, w, comms) + np.bincount(b, w, comms)
    inside = 2.0 * np.bincount(a[a == b], w[a == b], comms)
    two_w = strength.sum()
    return float(np.sum(inside / two_w - (strength / two_w) ** 2))
