"""Coarsening keys with and without their weight packed in."""
import numpy as np
import pytest

from test_gpu_parity import csr_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Louvain():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from louvaingpu_b200 import Louvain as L
    return L


@pytest.mark.parametrize("n,per", [(257, 3), (4099, 1), (20011, 40)])
@pytest.mark.parametrize("weights", [(0.0,), (1.0,), (0.0, 3.0, 4.0), (1.0, 2.0 ** 24), (2.0 ** 30, 5.0), (2.0 ** 31, 1.0),
                                     (2.0 ** 32, 7.0), (0.5, 1.0), (0.125, 2.0 ** 20)])
def test_coarse_list_of_any_weights(Louvain, oracle, gen, n, per, weights):
    """Whole weights up to the width left beside the community ids, wider ones,
    zeros (counted 1) and fractions: the oracle's coarse list and CSR.  Sums of
    these few distinct multiples of 1/8 are exact."""
    rng = np.random.default_rng(n)
    _, s, d, _ = gen.sbm(n, max(2, n // 200), 0.04, 2.0 / n, 1, 1, seed=n)
    pick = (np.minimum(s, d).astype(np.int64) * 7 + np.maximum(s, d)) % len(weights)
    w = np.array(weights, np.float32)[pick]
    comm = rng.integers(0, max(1, n // per), n).astype(np.int32)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        lv.set_communities(comm)
        part, C = lv.renumber()
        lv.induce()
        got = lv.level_edges()
        exp = oracle.induce(n, s, d, w, oracle.renumber(comm)[0])
        for x, y in zip(got, exp):
            np.testing.assert_array_equal(x, y)
        csr_equal(lv, oracle.Csr(C, *exp))
