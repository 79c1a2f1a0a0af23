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
