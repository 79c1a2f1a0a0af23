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
