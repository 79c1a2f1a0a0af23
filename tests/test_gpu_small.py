"""Runs of small graphs in one launch, against the oracle and the level kernels.

Weights are multiples of 1/8 throughout, so every sum is exact and results
are equal bit for bit, whichever path a level takes.
"""
import numpy as np
import pytest

from conftest import undirected_to_lists
from test_gpu_parity import csr_equal, make_case, run_equal, sorted_symmetric

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Louvain():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from louvaingpu_b200 import Louvain as L
    return L


def in_order(n, s, d, w):
    o = np.lexsort((d, s))
    return n, s[o], d[o], w[o]


def graph(gen, oracle, name):
    kind, _, arg = name.partition(":")
    if kind == "star":          # one row of `arg` entries: at the tile's length, one above it, far above it
        k = int(arg)
        s, d, w = undirected_to_lists([(0, i) for i in range(1, k + 1)] + [(1, 2)])
        return in_order(k + 1, s, d, w)
    if kind == "stars8":        # the same with weights in eighths (FP64 tiles hold 2048 entries)
        n, s, d, w = graph(gen, oracle, "star:" + arg)
        return n, s, d, (w * 0.125).astype(np.float32)
    if kind == "isolated":      # a few entries among 65,536 vertices, or one more than the path takes
        n = int(arg)
        return in_order(n, *undirected_to_lists([(0, n - 1), (0, 7), (7, n - 1), (7, 9), (40000, 40001)]))
    if kind == "one":
        return 2, np.array([0, 1], np.int32), np.array([1, 0], np.int32), np.ones(2, np.float32)
    if kind == "loop":          # a self loop alone
        return 3, np.array([1], np.int32), np.array([1], np.int32), np.ones(1, np.float32)
    if kind == "case":          # zero weights, self loops, isolated vertices
        n, s, d, w = make_case(gen, arg)
        return (n, *sorted_symmetric(oracle, n, s, d, w))
    if kind == "eighths":
        n, s, d, w = gen.sbm(int(arg), max(2, int(arg) // 50), 0.15, 2.0 / int(arg), 1, 9, seed=5)
        return n, s, d, (w * 0.125).astype(np.float32)
    if kind == "heavy":         # degrees above 2^30: no 32-bit sums
        n, s, d, w = gen.sbm(300, 6, 0.3, 0.01, 1, 1, seed=6)
        return n, s, d, (w * np.float32(2.0 ** 28)).astype(np.float32)
    if kind == "dense":         # rows of n - 1 entries, all in one community
        n = int(arg)
        s, d = np.divmod(np.arange(n * n, dtype=np.int32), np.int32(n))
        return n, s[s != d], d[s != d], np.ones(n * n - n, np.float32)
    if kind == "gaps":          # cliques with runs of vertices without edges between them, more than a block records
        size, gap, count = map(int, arg.split(":"))
        i, j = np.divmod(np.arange(size * size), size)
        at = (np.arange(count) * (size + gap))[:, None]
        s, d = ((at + x[i != j]).ravel().astype(np.int32) for x in (i, j))
        return count * (size + gap), s, d, np.ones(len(s), np.float32)
    n = int(arg)                # sbm:<n>
    return gen.sbm(n, max(2, n // 60), 0.25, 3.0 / n, 1, 4, seed=n)


NAMES = ["one:", "loop:", "star:4095", "star:4096", "star:4097", "star:9000", "star:66000", "stars8:2048", "stars8:2049",
         "isolated:65536", "isolated:65537", "case:loops_zeros_isolated", "case:odd_sizes", "case:weighted",
         "eighths:900", "eighths:4001", "heavy:", "dense:64", "dense:511", "dense:513", "sbm:70", "sbm:1025",
         "sbm:2049", "sbm:8193", "sbm:14001", "gaps:15:66:70", "gaps:100:200:60"]


@pytest.mark.parametrize("name", NAMES)
def test_run_equals_the_oracle(Louvain, oracle, gen, name):
    n, s, d, w = graph(gen, oracle, name)
    orun = oracle.Run(n, s, d, w)
    with Louvain() as lv:
        for _ in range(2):      # a second run starts from the list again
            lv.load_edges(s, d, w, n)
            run_equal(lv, lv.run(), orun, n, s, d, w, oracle)
            run_equal(lv, lv.run(), orun, n, s, d, w, oracle)


@pytest.mark.parametrize("name", ["sbm:1025", "eighths:900", "star:4097", "star:9000", "case:loops_zeros_isolated"])
def test_calls_after_a_run_see_its_last_level(Louvain, oracle, gen, name):
    """The last level's CSR, Q and list, its coarsening, and a step-by-step
    run on the same load, after a run that built none of its levels."""
    n, s, d, w = graph(gen, oracle, name)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        csr_equal(lv, oracle.Csr(n, s, d, w))
        res = lv.run()
        last = lv.level_info(res.n_levels - 1)
        assert lv.modularity() == last.q_level
        es, ed, ew = lv.level_edges()
        assert len(es) == last.n_entries
        csr_equal(lv, oracle.Csr(last.n_vertices, es, ed, ew))
        part = lv.level_partition(res.n_levels - 1)
        lv.induce()
        for got, exp in zip(lv.level_edges(), oracle.induce(last.n_vertices, es, ed, ew, part)):
            np.testing.assert_array_equal(got, exp)
        final = lv.partition()
        assert lv.run() == res
        np.testing.assert_array_equal(lv.partition(), final)


@pytest.mark.parametrize("kw", [dict(max_passes=1), dict(max_levels=1), dict(max_levels=2), dict(level_min_gain=0.2)])
def test_caps_and_thresholds(Louvain, oracle, gen, kw):
    """Runs stopped early end as the level kernels end them (an unsorted list
    takes those from level 0 on)."""
    n, s, d, w = gen.sbm(3000, 30, 0.05, 0.002, 1, 4, seed=2)
    mix = np.random.default_rng(1).permutation(len(s))
    out = []
    for o in (slice(None), mix):
        with Louvain(**kw) as lv:
            lv.load_edges(s[o], d[o], w[o], n)
            try:
                lv.run()
                status = 0
            except Exception as e:
                status = e.status
            out.append((status, lv.n_levels, lv.partition().tolist(),
                        [(lv.level_info(k).q_level, lv.level_info(k).passes) for k in range(lv.n_levels)]))
    assert out[0] == out[1]


@pytest.mark.parametrize("n,comms,p_in", [(30011, 150, 0.06), (90001, 450, 0.06), (200003, 900, 0.05), (240003, 600, 0.05)])
def test_larger_graphs(Louvain, oracle, gen, n, comms, p_in):
    """A cooperative grid for the whole run (coarse keys of 32 and of 64 bits),
    and for the last levels of a run whose first are too large for it."""
    n, s, d, w = gen.sbm(n, comms, p_in, 2.0 / n, 1, 3, seed=9)
    assert (len(s) > 64 * 1024) and ((len(s) > 4 * 1024 * 1024) == (n > 240000))
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        run_equal(lv, lv.run(), oracle.Run(n, s, d, w), n, s, d, w, oracle)
        run_equal(lv, lv.run(), oracle.Run(n, s, d, w), n, s, d, w, oracle)


@pytest.mark.parametrize("kind", ["sbm:9001", "sbm:30011", "linked:70001", "hub:60001"])
@pytest.mark.parametrize("scale", [1.0, 0.125])
def test_coarse_lists_in_one_direction(Louvain, oracle, gen, kind, scale):
    """Edges listed once, in any order: coarse lists are sorted but not
    symmetric (of more vertices than 16 bits hold, or with a row longer than a
    tile, for the linked triangles)."""
    rng = np.random.default_rng(8)
    n = int(kind.split(":")[1])
    if kind.startswith("sbm"):
        _, s, d, w = gen.sbm(n, n // 60, 0.25, 3.0 / n, 1, 4, seed=n)
        up = s <= d
        s, d, w = s[up], d[up], w[up]
    else:                       # triangles, linked at random, or all to the first
        t = np.arange(n, dtype=np.int32) * 3
        other = t[rng.integers(0, n, n)] if kind.startswith("linked") else np.zeros(n, np.int32)
        s = np.concatenate([t, t, t + 1, t[1:], t[::5]])
        d = np.concatenate([t + 1, t + 2, t + 2, other[1:], t[::5]])
        w = np.concatenate([np.full(3 * n, 8), np.ones(n - 1), np.full(len(t[::5]), 2)]).astype(np.float32)
        n = 3 * n
    o = rng.permutation(len(s))
    s, d, w = s[o], d[o], (w[o] * np.float32(scale)).astype(np.float32)
    flip = rng.random(len(s)) < 0.5
    s, d = np.where(flip, d, s), np.where(flip, s, d)
    orun = oracle.Run(n, s, d, w)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        run_equal(lv, lv.run(), orun, n, s, d, w, oracle)
        run_equal(lv, lv.run(), orun, n, s, d, w, oracle)


def test_batch_mixes_the_paths(Louvain, oracle, gen):
    """Graphs for clusters of 1, 2, 4 and 8 blocks, ones the launch leaves
    open (unsorted, a row too long), larger ones, and one without entries:
    each as run alone."""
    graphs = [graph(gen, oracle, x) for x in NAMES]
    graphs.append((5, np.zeros(0, np.int32), np.zeros(0, np.int32), np.zeros(0, np.float32)))
    n, s, d, w = gen.sbm(2000, 20, 0.05, 0.002, 1, 4, seed=2)
    o = np.random.default_rng(3).permutation(len(s))
    graphs += [(n, s[o], d[o], w[o]), gen.sbm(60001, 300, 0.06, 0.00005, 1, 3, seed=9)]
    with Louvain() as lv:
        b = lv.run_batch(graphs)
        for g, (n, s, d, w) in enumerate(graphs):
            lv.load_edges(s, d, w, n)
            res = lv.run()
            assert (b.n_levels[g], b.n_comms[g], b.status[g]) == (res.n_levels, res.n_comms, 0), g
            np.testing.assert_array_equal(b.part(g), lv.partition(), err_msg=str(g))
            assert b.q_final[g] == pytest.approx(res.q_final, abs=1e-12), g
