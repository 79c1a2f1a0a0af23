"""Batched runs at the sizes where the batch kernels change their path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Louvain():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from louvaingpu_b200 import Louvain as L
    return L


def cycle(n, w=1.0):
    """Both directions of a cycle on n >= 3 vertices, sorted by (src, dst)."""
    e = sorted({(i, (i + d) % n) for i in range(n) for d in (1, -1)})
    s, d = np.array(e, np.int32).T.copy()
    return n, s, d, np.full(len(s), w, np.float32)


def same_as_single(Louvain, graphs):
    with Louvain() as lv:
        b = lv.run_batch(graphs)
    with Louvain() as lv:
        for g, (n, s, d, w) in enumerate(graphs):
            lv.load_edges(s, d, w, n)
            res = lv.run()
            assert b.q_final[g] == res.q_final, g
            assert (b.n_levels[g], b.n_comms[g], b.status[g]) == (res.n_levels, res.n_comms, 0), g
            np.testing.assert_array_equal(b.part(g), lv.partition(), err_msg=str(g))


@pytest.mark.parametrize("sizes", [(1024, 1024, 1024), (1023, 1025, 3, 1024), (3,) * 700, (2048, 3, 4096, 5000)])
def test_graph_boundaries_around_the_sum_tiles(Louvain, sizes):
    """m and the entry counts are summed in tiles of 2048 entries (a cycle on
    n vertices has 2n): boundaries on, beside and many inside a tile.
    Integral weights: every sum is exact, so results are equal bit for bit."""
    same_as_single(Louvain, [cycle(n, 1.0 + k % 3) for k, n in enumerate(sizes)])


@pytest.mark.parametrize("scale", [1.0, 0.125])
def test_coarsening_methods_agree_while_graphs_finish_at_different_levels(Louvain, gen, scale):
    """The batch coarsens by transposition with the finished graphs' rows left
    out, or by sorting all keys (coarsen_mode 3): the same results, graph by
    graph.  Weights are multiples of 1/8, so every sum is exact."""
    graphs = [cycle(3), cycle(17), (4, np.zeros(0, np.int32), np.zeros(0, np.int32), np.zeros(0, np.float32))]
    for k, n in enumerate((70, 500, 3001, 9000)):
        n, s, d, w = gen.sbm(n, max(2, n // 40), 0.2, 3.0 / n, 1, 4, seed=k)
        graphs.append((n, s, d, (w * scale).astype(np.float32)))
    out = []
    for mode in (0, 3):
        with Louvain(coarsen_mode=mode) as lv:
            out.append(lv.run_batch(graphs))
    a, b = out
    assert len(set(a.n_levels.tolist())) > 1
    np.testing.assert_array_equal(a.partition, b.partition)
    np.testing.assert_array_equal(a.n_levels, b.n_levels)
    np.testing.assert_array_equal(a.q_final, b.q_final)
    same_as_single(Louvain, graphs)
