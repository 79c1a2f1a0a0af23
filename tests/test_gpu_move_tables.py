"""Decisions of a hashing pass where the shared-memory tables can go wrong."""
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


def rows_graph(degrees, n, scale, seed):
    """Vertex i < len(degrees) with degrees[i] distinct neighbours at the upper
    end of 0..n-1, both directions, weights k * scale."""
    rng = np.random.default_rng(seed)
    s = np.repeat(np.arange(len(degrees), dtype=np.int32), degrees)
    d = np.concatenate([len(degrees) + rng.permutation(n - len(degrees))[:k] for k in degrees]).astype(np.int32)
    w = (rng.integers(1, 5, len(s)) * scale).astype(np.float32)
    s, d, w = np.r_[s, d], np.r_[d, s], np.r_[w, w]
    o = np.lexsort((d, s))
    return n, s[o], d[o], w[o]


@pytest.mark.parametrize("scale", [1.0, 0.125])
@pytest.mark.parametrize("kind", ["own", "few", "one", "ties"])
@pytest.mark.parametrize("degrees", [(33, 34, 512, 511, 33), (512,) * 9, (513, 1024, 1025, 2049), (4097, 5000, 9001)])
def test_decisions_for_rows_at_the_class_edges(Louvain, oracle, degrees, kind, scale):
    """Rows at the edges of the tile, block and hub classes over communities
    of their own, a few, one only, and many with equal gains (the lowest id
    wins): the oracle's decisions exactly (weights in eighths: exact sums)."""
    n, s, d, w = rows_graph(degrees, 12000, scale, 4)
    if kind == "ties":
        w[:] = scale
    rng = np.random.default_rng(5)
    first = len(degrees)
    comm = np.arange(n, dtype=np.int32)
    if kind == "few":
        comm[first:] = first + rng.integers(0, 7, n - first)
    elif kind == "one":
        comm[first:] = n - 1
    elif kind == "ties":
        comm[first:] = first + (np.arange(n - first) // 2)
    c = oracle.Csr(n, s, d, w)
    tot, size = np.zeros(n), np.zeros(n, np.int32)
    np.add.at(tot, comm, c.k)
    np.add.at(size, comm, 1)
    with Louvain() as lv:
        lv.load_edges(s, d, w, n)
        lv.set_communities(comm)
        nxt, cand = lv.move_decide()
    exp_nxt, exp_cand, _ = c.decide(comm, tot, size)
    np.testing.assert_array_equal(nxt, exp_nxt)
    np.testing.assert_array_equal(cand, exp_cand)
