"""Small runs at the edges of what they take: weights, sizes, memory, waits.

Against the oracle, and the calls that follow a run against the run itself.
"""
import numpy as np
import pytest

from conftest import undirected_to_lists
from test_gpu_parity import run_equal
from test_gpu_small import in_order

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Louvain():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from louvaingpu_b200 import Louvain as L
    return L


def triangles():
    """Two triangles joined by an edge."""
    return in_order(6, *undirected_to_lists([(0, 1), (1, 2), (0, 2), (3, 4), (4, 5), (3, 5), (2, 3)]))


@pytest.mark.parametrize("unit", [2e18, 2.0 ** 62, 1e20, 2.0 ** 70, 1e30])
def test_whole_weights_beyond_integers(Louvain, oracle, gen, unit):
    """Whole weights whose sums, or which themselves, do not fit 63 bits: a
    coarse list of few communities in shared memory sums them in FP64.  The
    weights of a graph lie within a factor of four, so every sum is exact."""
    graphs = [triangles(), gen.sbm(300, 6, 0.3, 0.01, 1, 4, seed=6), gen.sbm(500, 80, 0.9, 0.01, 1, 4, seed=7)]
    graphs = [(n, s, d, (w * np.float32(unit)).astype(np.float32)) for n, s, d, w in graphs]
    with Louvain() as lv:
        b = lv.run_batch(graphs)
        for g, (n, s, d, w) in enumerate(graphs):
            orun = oracle.Run(n, s, d, w)
            lv.load_edges(s, d, w, n)
            run_equal(lv, lv.run(), orun, n, s, d, w, oracle)
            np.testing.assert_array_equal(b.part(g), orun.final)
            assert b.n_levels[g] == len(orun.levels)


def listed_once(n, degree, seed):
    """A graph of 50-vertex blocks, every edge listed once, in any order."""
    rng = np.random.default_rng(seed)
    s = rng.integers(0, n, n * degree)
    d = np.where(rng.random(len(s)) < 0.8, s // 50 * 50 + rng.integers(0, 50, len(s)), rng.integers(0, n, len(s)))
    d = np.minimum(d, n - 1)
    keep = s != d
    return n, s[keep].astype(np.int32), d[keep].astype(np.int32), rng.integers(1, 5, keep.sum()).astype(np.float32)


@pytest.fixture(scope="module")
def unsorted_graphs():
    """6.3 M entries in graphs a cluster starts and leaves open."""
    return [listed_once(5000, 10, k) for k in range(128)]


def check_sample(oracle, graphs, part, n_levels, sample=(0, 31, 64, 127)):
    for g in sample:
        orun = oracle.Run(*graphs[g])
        np.testing.assert_array_equal(part(g), orun.final, err_msg=str(g))
        assert n_levels[g] == len(orun.levels)


@pytest.mark.parametrize("others", [0, 1])
@pytest.mark.parametrize("where", ["host", "device"])
def test_batches_of_unsorted_small_graphs_fit_the_default_arena(Louvain, oracle, gen, unsorted_graphs, where, others):
    """The union that takes the graphs left open needs the memory they were
    started in, and the staged copies of host lists.  others: beside a graph
    that is no small run, and ones that are and finish."""
    graphs = list(unsorted_graphs)
    if others:
        graphs += [gen.sbm(40000, 200, 0.06, 2.0 / 40000, 1, 4, seed=1), gen.sbm(900, 20, 0.3, 0.01, 1, 4, seed=2)]
    with Louvain() as lv:
        if where == "host":
            b = lv.run_batch(graphs)
        else:
            import torch
            from louvaingpu_b200.louvain import pack_graphs
            s, d, w, eoff, voff = pack_graphs(graphs)
            t = [torch.from_numpy(x).cuda() for x in (s, d, w)]
            torch.cuda.synchronize()
            b = lv.run_batch_device(*(x.data_ptr() for x in t), eoff, voff)
    assert not b.status.any()
    check_sample(oracle, graphs, b.part, b.n_levels, (0, 31, 64, 127) + tuple(range(128, len(graphs))))


def test_server_groups_of_unsorted_small_graphs_stay_whole(oracle, unsorted_graphs):
    """A slot of just the footprint of all requests runs them as one group (a
    group that exhausts the arena would be split in two)."""
    import ctypes
    import torch
    from louvaingpu_b200 import _lib
    from louvaingpu_b200.serving import Server
    graphs = unsorted_graphs
    t = [[torch.from_numpy(x).cuda() for x in g[1:]] for g in graphs]
    torch.cuda.synchronize()
    E, V, size = sum(len(g[1]) for g in graphs), sum(g[0] for g in graphs), ctypes.c_int64()
    assert _lib.load().lvg_batch_footprint(V, E, len(graphs), ctypes.byref(size)) == 0
    parts = [np.zeros(g[0], np.int32) for g in graphs]
    with Server(n_slots=1, hbm_budget=size.value, max_batch_entries=E, max_batch_graphs=len(graphs)) as srv:
        ids = [srv.submit(*(x.data_ptr() for x in a), len(g[1]), g[0], part_out=p)
               for a, g, p in zip(t, graphs, parts)]
        srv.drain(timeout_ms=60000)
        got = {r.id: r for r in srv.poll(len(graphs))}
        taken = srv.stats()["batches"]
    assert all(got[i].status == 0 for i in ids)
    sizes = [got[i].batch_graphs for i in ids]
    assert sum(sizes.count(k) // k for k in set(sizes)) == taken   # groups as the slot took them
    check_sample(oracle, graphs, lambda g: parts[g], [got[i].n_levels for i in ids])


@pytest.mark.parametrize("max_levels", [1, 2, -1])
@pytest.mark.parametrize("n,blocks", [(60, 4), (400, 12), (3001, 60), (30011, 300), (90001, 450)])
def test_state_after_a_run_is_the_runs_own(Louvain, gen, n, blocks, max_levels):
    """Weights over 60 binary orders, so that sums depend on their order: Q
    and labels that a call after the run sees are those the run ended in, not
    those of its passes run again."""
    from louvaingpu_b200 import LvgError
    n, s, d, _ = gen.sbm(n, blocks, min(0.5, 15.0 * blocks / n), 2.0 / n, 1, 1, seed=n)
    for seed in range(4):
        x = np.random.default_rng(seed).random(n) * 30.0
        w = np.exp2(x[s] + x[d] - 30.0).astype(np.float32)
        with Louvain(max_levels=max_levels) as lv:
            lv.load_edges(s, d, w, n)
            try:
                lv.run()
            except LvgError as e:
                assert e.status == 4 and max_levels > 0   # the level cap
            last = lv.n_levels - 1
            labels, part, info = lv.level_labels(last), lv.level_partition(last), lv.level_info(last)
            assert lv.modularity() == info.q_level
            again, comms = lv.renumber()
            np.testing.assert_array_equal(again, part)
            assert comms == info.n_comms
            np.testing.assert_array_equal(lv.level_labels(last + 1), labels)


@pytest.mark.parametrize("fault", ["id", "weight"])
def test_a_refused_batch_writes_nothing(gen, fault):
    """A bad entry of a small graph is found beside the union of the others:
    the call is refused with every output as it was."""
    from louvaingpu_b200 import _lib, Louvain
    from louvaingpu_b200.louvain import pack_graphs
    bad = gen.sbm(500, 10, 0.3, 0.01, 1, 4, seed=3)
    if fault == "id":
        bad[2][-1] = 500
    else:
        bad[3][7] = -1.0
    graphs = [gen.sbm(60001, 300, 0.06, 0.00005, 1, 3, seed=9), gen.sbm(900, 20, 0.3, 0.01, 1, 4, seed=2), bad]
    s, d, w, eoff, voff = pack_graphs(graphs)
    p = lambda x: x.ctypes.data
    outs = [np.full(voff[-1], -7, np.int32), np.full(3, -7.0), *(np.full(3, -7, np.int32) for _ in range(3))]
    L = _lib.load()
    with Louvain(arena_bytes=1 << 30) as lv:   # room for both at once
        assert L.lvg_batch_run(lv._h, p(s), p(d), p(w), p(eoff), p(voff), 3, *map(p, outs)) == 1
        assert all((x == -7).all() for x in outs)
        b = lv.run_batch(graphs[:2])
        assert not b.status.any()


def test_a_build_after_the_load_reads_no_facts_again(Louvain, oracle, gen):
    """A list that waits with its build keeps what the load learnt of it: the
    launches up to Q are those of a load that builds at once (as it does in an
    arena without room for any list's build)."""
    import ctypes
    from louvaingpu_b200 import _lib
    from test_gpu_parity import csr_equal
    n, s, d, w = gen.sbm(3001, 60, 0.2, 0.001, 1, 4, seed=1)
    L, counts = _lib.load(), []
    for arena in (0, 24 << 20):
        with Louvain(arena_bytes=arena) as lv:
            lv.load_edges(s, d, w, n)          # (the first sizes the arena)
            at = [ctypes.c_int64(), ctypes.c_int64()]
            L.lvg_kernel_launches(ctypes.byref(at[0]))
            lv.load_edges(s, d, w, n)
            lv.modularity()
            L.lvg_kernel_launches(ctypes.byref(at[1]))
            counts.append(at[1].value - at[0].value)
            csr_equal(lv, oracle.Csr(n, s, d, w))
    assert counts[0] == counts[1]


@pytest.fixture
def hooks():
    from louvaingpu_b200 import _lib
    L = _lib.load()
    yield L
    assert L.lvg_debug_small_launch(0) == 0 and L.lvg_debug_small_hold(-1, 0) == 0


def launches():
    import ctypes
    from louvaingpu_b200 import _lib
    n = ctypes.c_int64()
    _lib.load().lvg_kernel_launches(ctypes.byref(n))
    return n.value


def run_counted(lv):
    n = launches()
    res = lv.run()
    return res, launches() - n


# n, blocks: a cluster's list; a grid's; a grid's behind levels of the level
# kernels, as the list is in no order
@pytest.mark.parametrize("n,blocks,unsorted", [(2000, 40, False), (30011, 300, False), (30011, 300, True)])
@pytest.mark.parametrize("error", [720, 912, 701, 9, 801])
def test_a_refused_launch_leaves_the_run_to_the_level_kernels(Louvain, oracle, gen, hooks, n, blocks, unsorted, error):
    n, s, d, w = gen.sbm(n, blocks, 15.0 * blocks / n, 2.0 / n, 1, 4, seed=5)
    if unsorted:
        o = np.random.default_rng(2).permutation(len(s))
        s, d, w = s[o], d[o], w[o]
    orun = oracle.Run(n, s, d, w)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        ref, n_ref = run_counted(lv)
        run_equal(lv, ref, orun, n, s, d, w, oracle)
        lv.load_edges(s, d, w, n)          # (a second run would build level 0 again)
        assert hooks.lvg_debug_small_launch(error) == 0
        res, n_res = run_counted(lv)
        assert n_res > n_ref + 20
        run_equal(lv, res, orun, n, s, d, w, oracle)
        lv.modularity()
        b = lv.run_batch([(n, s, d, w), triangles()])
        np.testing.assert_array_equal(b.part(0), orun.final)
        assert hooks.lvg_debug_small_launch(0) == 0
        lv.load_edges(s, d, w, n)
        assert run_counted(lv) == (ref, n_ref)


def test_other_launch_errors_are_reported(Louvain, gen, hooks):
    from louvaingpu_b200 import LvgError
    n, s, d, w = gen.sbm(2000, 40, 0.3, 0.001, 1, 4, seed=5)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        ref = lv.run()
        assert hooks.lvg_debug_small_launch(999) == 0
        for call in (lv.run, lambda: lv.run_batch([(n, s, d, w)])):
            with pytest.raises(LvgError) as e:
                call()
            assert e.value.status == 5
        assert hooks.lvg_debug_small_launch(0) == 0
        lv.load_edges(s, d, w, n)
        assert lv.run() == ref


@pytest.mark.parametrize("unsorted", [False, True])
def test_a_grid_wait_runs_out(Louvain, oracle, gen, hooks, unsorted):
    """A block that never comes to the grid's barriers: the others give up
    after 20 ms and the level kernels run instead."""
    n, s, d, w = gen.sbm(30011, 300, 0.15, 2.0 / 30011, 1, 4, seed=5)
    if unsorted:
        o = np.random.default_rng(2).permutation(len(s))
        s, d, w = s[o], d[o], w[o]
    orun = oracle.Run(n, s, d, w)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        ref, n_ref = run_counted(lv)
        for block in (0, 1):
            lv.load_edges(s, d, w, n)      # (a second run would build level 0 again)
            assert hooks.lvg_debug_small_hold(block, 20_000_000) == 0
            res, n_res = run_counted(lv)
            assert n_res > n_ref + 20
            run_equal(lv, res, orun, n, s, d, w, oracle)
        assert hooks.lvg_debug_small_hold(-1, 0) == 0
        lv.load_edges(s, d, w, n)
        assert run_counted(lv) == (ref, n_ref)


def test_thousands_of_tiny_graphs_run_by_clusters(Louvain, oracle):
    """Their memory is a few KB each, so a default arena holds them all: one
    launch of the levels and three behind it, not a union's."""
    from test_gpu_batch_edges import cycle
    graphs = [cycle(3 + k % 60, 1.0 + k % 5) for k in range(3000)]
    with Louvain() as lv:
        lv.run_batch(graphs)
        n = launches()
        b = lv.run_batch(graphs)
        assert launches() - n <= 8
    check_sample(oracle, graphs, b.part, b.n_levels, range(0, 3000, 97))


@pytest.mark.parametrize("n,blocks", [(300, 6), (2000, 40), (30011, 300)])
@pytest.mark.parametrize("max_passes", [1, 2, 5, 40])
def test_every_pass_of_the_last_level_has_its_time(Louvain, gen, n, blocks, max_passes):
    """A gain below the threshold never ends this level: it takes all passes
    it may (by one block, a cluster, a grid)."""
    from louvaingpu_b200 import LvgError
    n, s, d, w = gen.sbm(n, blocks, 15.0 * blocks / n, 2.0 / n, 1, 4, seed=5)
    with Louvain(pass_min_gain=-2.0, max_passes=max_passes) as lv:
        lv.load_edges(s, d, w, n)
        with pytest.raises(LvgError) as e:
            lv.run()
        assert e.value.status == 4 and lv.n_levels == 1 and lv.level_info(0).passes == max_passes
        times = lv.move_pass_times()
        total, passes = lv.move_stats()
    assert len(times) == passes == max_passes
    assert all(t > 0 for t in times) and total == pytest.approx(sum(times), rel=1e-5)


def sized(n, entries, seed=0):
    """A sorted symmetric list of exactly `entries` entries on n vertices in
    blocks of 64 (an odd number has a self loop)."""
    rng, pairs = np.random.default_rng(seed), entries // 2
    at = np.zeros(0, np.int64)
    while len(at) < pairs:
        a = rng.integers(0, n, 2 * pairs)
        b = np.where(rng.random(len(a)) < 0.7, a // 64 * 64 + rng.integers(0, 64, len(a)), rng.integers(0, n, len(a)))
        b = np.minimum(b, n - 1)
        at = np.union1d(at, (np.minimum(a, b) * n + np.maximum(a, b))[a != b])
    a, b = np.divmod(rng.permutation(at)[:pairs], n)
    w = rng.integers(1, 5, pairs)
    loop = [n // 2] if entries % 2 else []
    s, d, w = np.concatenate([a, b, loop]), np.concatenate([b, a, loop]), np.concatenate([w, w, [3] * len(loop)])
    return in_order(n, s.astype(np.int32), d.astype(np.int32), w.astype(np.float32))


MAX_V, MAX_E, CLUSTER, RESIDENT = 1 << 18, 1 << 22, 1 << 16, (512, 6144)


@pytest.mark.parametrize("make,small", [
    (lambda: sized(MAX_V, 1500000), True), (lambda: sized(MAX_V + 1, 1500000), False),
    (lambda: sized(MAX_V, 20000), True), (lambda: sized(MAX_V + 1, 20000), False),
    (lambda: sized(90000, MAX_E), True), (lambda: sized(90000, MAX_E + 1), False),
    (lambda: sized(15536, CLUSTER - 15536), True), (lambda: sized(15536, CLUSTER - 15535), True),
    (lambda: sized(*RESIDENT), True), (lambda: sized(RESIDENT[0] + 1, RESIDENT[1]), True),
    (lambda: sized(RESIDENT[0], RESIDENT[1] + 1), True)],
    ids=["V", "V+1", "sparse_V", "sparse_V+1", "E", "E+1", "cluster", "grid", "block", "block_V+1", "block_E+1"])
def test_limits_of_a_run(Louvain, oracle, make, small):
    n, s, d, w = make()
    orun = oracle.Run(n, s, d, w)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        res, count = run_counted(lv)
        assert (count < 10) == small
        run_equal(lv, res, orun, n, s, d, w, oracle)
        assert lv.modularity() == lv.level_info(res.n_levels - 1).q_level


def test_limits_of_a_batch(Louvain, oracle):
    """Graphs at and one entry above the steps of the clusters' sizes, and of
    what a batch gives to clusters."""
    graphs = [sized(k // 12, k + more) for k in (16 << 10, 48 << 10, 128 << 10, 256 << 10) for more in (0, 1)]
    with Louvain(arena_bytes=1 << 30) as lv:
        b = lv.run_batch(graphs)
    check_sample(oracle, graphs, b.part, b.n_levels, range(len(graphs)))


@pytest.mark.parametrize("n", [200, 1000])
def test_runs_of_more_levels_than_a_launch_takes(Louvain, oracle, n):
    """A ring merges a few vertices a level: the launch leaves the run open
    (its levels' partitions, or records, are full) and the level kernels end it."""
    from test_gpu_batch_edges import cycle
    n, s, d, w = cycle(n)
    orun = oracle.Run(n, s, d, w)
    assert len(orun.levels) > 12
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        res, count = run_counted(lv)
        assert count > 100
        run_equal(lv, res, orun, n, s, d, w, oracle)
        b = lv.run_batch([(n, s, d, w), triangles()])
        np.testing.assert_array_equal(b.part(0), orun.final)
        assert b.n_levels[0] == len(orun.levels)


def accepted(make, n, s, d, w, arena):
    """Which of the calls of a session succeed in an arena."""
    from louvaingpu_b200 import LvgError
    out = []
    with make(arena_bytes=arena) as lv:
        for call in (lambda: lv.load_edges(s, d, w, n), lv.run, lv.modularity, lv.induce, lv.modularity, lv.run,
                     lambda: lv.modularity_fp64(np.zeros(n, np.int32))):
            try:
                call()
                out.append(True)
            except LvgError as e:
                assert e.status == 2 or (e.status == 6 and False in out)   # out of memory, or behind such a call
                out.append(False)
                if len(out) == 1:
                    break
    return out


@pytest.mark.parametrize("kind", ["once", "sorted"])
def test_tight_arenas_hold_what_the_level_kernels_do_there(Louvain, gen, kind):
    """Few edges among 200,000 vertices, where a small run's memory differs
    most: no call that succeeds by the level kernels is refused behind one."""
    _, s, d, w = listed_once(2000, 8, 2) if kind == "once" else gen.sbm(500, 10, 0.3, 0.01, 1, 4, seed=1)
    size, held = 30e6, 0
    while size < 72e6:
        level = accepted(lambda **kw: Louvain(level_kernels=True, **kw), 200000, s, d, w, int(size))
        small = accepted(Louvain, 200000, s, d, w, int(size))
        assert all(small[:len(level)][i] for i, ok in enumerate(level) if ok), (int(size), level, small)
        held += all(level)
        size *= 1.008
    assert held > 10
