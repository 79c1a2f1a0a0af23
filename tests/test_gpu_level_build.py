"""The two-pass level build at the sizes where its blocks and rows can go wrong."""
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


def path(n, loops=(), first=0):
    """A path on first..n-1 with self loops at `loops`, sorted and symmetric."""
    i = np.arange(first, n - 1, dtype=np.int32)
    lp = np.array(loops, np.int32)
    s, d = np.r_[i, i + 1, lp], np.r_[i + 1, i, lp]
    o = np.lexsort((d, s))
    return s[o], d[o], (1.0 + (s[o] + d[o]) % 3).astype(np.float32)


@pytest.mark.parametrize("chunk", [0, 4096])
@pytest.mark.parametrize("n,loops,first", [(3, (), 0), (1024, (), 0), (1025, (), 0), (1025, (0, 1, 1024), 0), (1026, (), 0),
                                           (9000, (0, 17, 8999), 0), (9000, (8999,), 8000), (20000, range(0, 20000, 3), 0)])
def test_csr_of_sorted_lists(Louvain, oracle, n, loops, first, chunk):
    """Lists of one entry less, exactly and more than whole 2048-entry blocks,
    with self loops at row starts and ends, empty leading and trailing rows,
    copied at once and in chunks: the oracle's CSR."""
    s, d, w = path(n, loops, first)
    with Louvain(load_chunk_entries=chunk) as lv:
        lv.load_edges(s, d, w, n + 5)
        csr_equal(lv, oracle.Csr(n + 5, s, d, w))


@pytest.mark.parametrize("at", [0, 2047, 2048, -1])
@pytest.mark.parametrize("what", ["order", "weight", "direction", "id", "negative"])
def test_what_the_first_pass_must_see(Louvain, oracle, at, what):
    """One entry that breaks the order, the symmetry or the entry rules, at the
    start, the end and a block boundary of a list of many blocks:
    rejected, or built as the oracle builds any list."""
    n = 70000
    s, d, w = (x.copy() for x in path(n))
    if what == "order":
        j = at if at >= 0 else len(s) - 2
        for x in (s, d, w):
            x[[j, j + 1]] = x[[j + 1, j]]
    elif what == "weight":
        w[at] += 1.0
    elif what == "direction":
        s, d, w = (np.delete(x, at % len(s)) for x in (s, d, w))
    elif what == "id":
        d[at] = n
    else:
        w[at] = -1.0
    with Louvain() as lv:
        if what in ("id", "negative"):
            with pytest.raises(Exception) as e:
                lv.load_edges(s, d, w, n)
            assert e.value.status == 1
        else:
            lv.load_edges(s, d, w, n)
            csr_equal(lv, oracle.Csr(n, s, d, w))
