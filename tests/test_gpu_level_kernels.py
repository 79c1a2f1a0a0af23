"""The level kernels on lists that a small run would take.

Tests of the level kernels' settings, of batches as one union and of runs
against the oracle, each once more in contexts that take the level kernels for
every list.
"""
import numpy as np
import pytest

from test_gpu_autotune import (rmat16, test_autotune_picks_a_measured_pair_and_keeps_results,  # noqa: F401
                               test_autotuned_batched_run_equals_default, test_thresholds_do_not_change_results)
from test_gpu_batch import (test_batch_caps_are_per_graph, test_batch_equals_single_runs,  # noqa: F401
                            test_batch_matches_oracle, test_batch_persistent_kernels_at_low_thresholds,
                            test_many_tiny_graphs)
from test_gpu_batch_edges import (cycle,  # noqa: F401
                                  test_coarsening_methods_agree_while_graphs_finish_at_different_levels,
                                  test_graph_boundaries_around_the_sum_tiles)
from test_gpu_parity import test_graph_replay_and_sync_interval_do_not_change_results  # noqa: F401
from test_gpu_small import test_run_equals_the_oracle  # noqa: F401
from test_gpu_small_limits import launches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Louvain():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from louvaingpu_b200 import Louvain as L
    return lambda **kw: L(level_kernels=True, **kw)


@pytest.mark.parametrize("batch", [False, True])
def test_the_setting_decides_the_path(Louvain, gen, batch):
    """A level of the level kernels takes some 40 launches, a small run five
    for all its levels; without that, the tests above compare nothing new."""
    from louvaingpu_b200 import Louvain as Either
    n, s, d, w = gen.sbm(3000, 30, 0.05, 0.002, 1, 4, seed=2)
    counts = []
    for make in (Either, Louvain):
        with make() as lv:
            lv.load_edges(s, d, w, n)
            at = launches()
            levels = lv.run_batch([(n, s, d, w)]).n_levels[0] if batch else lv.run().n_levels
            counts.append((launches() - at) / levels)
    assert counts[0] < 8 and counts[1] > 20


@pytest.mark.parametrize("modes", [(0, 1), (2, 3)])
def test_transposition_with_finished_graphs_left_out(Louvain, oracle, gen, modes):
    """Coarsening methods on a union whose graphs finish at different levels,
    against the oracle: by transposition (0, 2), by chunks or a sort of all keys."""
    graphs = [cycle(3), cycle(17), (4, np.zeros(0, np.int32), np.zeros(0, np.int32), np.zeros(0, np.float32))]
    graphs += [gen.sbm(n, max(2, n // 40), 0.2, 3.0 / n, 1, 4, seed=k) for k, n in enumerate((70, 500, 3001, 9000, 20011))]
    runs = [oracle.Run(*g) if len(g[1]) else None for g in graphs]
    assert len({len(r.levels) for r in runs if r}) > 1
    for mode in modes:
        with Louvain(coarsen_mode=mode) as lv:
            b = lv.run_batch(graphs)
        for g, r in enumerate(runs):
            np.testing.assert_array_equal(b.part(g), r.final if r else np.arange(4), err_msg=str(g))
            assert b.n_levels[g] == (len(r.levels) if r else 1), g
